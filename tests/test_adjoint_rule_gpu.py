"""The rule between the tangent pass and the backward sweep of the Heston
pathwise Greeks: a share in the money of 0.16 - 425 / (paths an SM) from 7,000
paths an SM on, 0.01 from 3,500."""
import math

import pytest

from openferric_b200 import _abi as A
from openferric_b200._lib import context
from openferric_b200.adjoint import HestonAdjointSpec, heston_adjoint

pytestmark = pytest.mark.gpu

BASE = dict(spot=100.0, rate=0.03, v0=0.04, kappa=2.0, theta=0.04, xi=0.5, rho=-0.7)


def _strike(share, asian, T=1.0):
    """The call strike that a share of the lognormal stand-in ends above."""
    mu = BASE["rate"] * T
    w = BASE["theta"] * T / (3.0 if asian else 1.0)
    f = math.log(math.expm1(mu) / mu) if asian else mu
    lo, hi = 0.0, 5.0
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if 0.5 * math.erfc(mid / math.sqrt(2.0)) > share else (lo, mid)
    return 100.0 * math.exp(f - 0.5 * w + lo * math.sqrt(w))


@pytest.mark.parametrize("asian", [False, True])
@pytest.mark.parametrize("per_sm,steps", [(3600, 33), (7100, 33), (30_000, 33), (3600, 2048), (7100, 2048)])
def test_both_sides_of_the_rule_agree(asian, per_sm, steps):
    """Strikes 1e-6 apart on the two sides of the rule: the same paths, 1e-5 of
    whose in-the-money ones change sides.  Either pass is within 1e-3 (2e-4
    absolute) of the FP64 difference, so within twice that of the other; at 2,048
    steps, the longest path, both share what the FP32 path itself is off."""
    paths = per_sm * context(0).sm_count
    K = _strike(0.16 - 425.0 / per_sm if per_sm >= 7000 else 0.01, asian)
    a, b = (heston_adjoint(HestonAdjointSpec(strike=K * x, expiry=1.0, num_paths=paths, num_steps=steps, seed=3,
                                             asian=asian), **BASE) for x in (1.0 - 5e-7, 1.0 + 5e-7))
    assert a.price == pytest.approx(b.price, rel=1e-4)
    for name in A.OF_ADJ_NAMES:
        assert abs(a.greeks[name] - b.greeks[name]) <= 2.0 * max(1e-3 * abs(b.greeks[name]), 2e-4), name


def test_many_paths_take_the_sweep_up_to_a_larger_share():
    """28,000 paths an SM, 128 steps: the sweep takes 0.91 of the tangent pass's
    time at a share of 0.125; the tangent pass's does not depend on the share."""
    paths = 28_000 * context(0).sm_count
    few, many = (min(heston_adjoint(HestonAdjointSpec(strike=_strike(s, True), expiry=1.0, num_paths=paths,
                                                      num_steps=128, seed=3, asian=True), **BASE).kernel_ms
                     for _ in range(6)) for s in (0.125, 0.25))
    assert few < 0.96 * many
