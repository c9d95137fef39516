"""The two ways to the Heston pathwise Greeks (of_heston_price_adjoint): the
pass that carries the derivatives along with the path, and the checkpointed
backward sweep taken where fewer than a tenth of at least 7,000 paths an SM
are expected in the money."""
import math

import pytest

from openferric_b200 import OptionType
from openferric_b200 import _abi as A
from openferric_b200.adjoint import HestonAdjointSpec, heston_adjoint

pytestmark = pytest.mark.gpu

BASE = dict(spot=100.0, rate=0.03, v0=0.04, kappa=2.0, theta=0.04, xi=0.5, rho=-0.7)


def _fd(spec, name, bump=1e-6):  # few paths: a wider bump takes some of them across a kink of the step
    h = bump * abs(BASE[name])
    up, dn = dict(BASE), dict(BASE)
    up[name] += h
    dn[name] -= h
    return (heston_adjoint(spec, forward_only=2, **up).price - heston_adjoint(spec, forward_only=2, **dn).price) / (2 * h)


@pytest.mark.parametrize("asian", [False, True])
@pytest.mark.parametrize("steps", [1, 2, 3, 33, 512])
def test_tangents_match_central_differences_at_the_edges_of_a_path(steps, asian):
    """Odd and smallest step counts and the largest in use, a path count that fills no warp:
    the tolerance is that of the 2^20-path comparison (1e-3 of the difference,
    2e-4 absolute), a put in the money so that few paths cross the kink."""
    spec = HestonAdjointSpec(strike=140.0, expiry=1.0, num_paths=16385, num_steps=steps, seed=5, asian=asian,
                             option_type=OptionType.Put)
    res = heston_adjoint(spec, **BASE)
    assert res.price == heston_adjoint(spec, forward_only=1, **BASE).price
    for name in A.OF_ADJ_NAMES:
        fd = _fd(spec, name)
        assert abs(res.greeks[name] - fd) <= max(1e-3 * abs(fd), 2e-4), (name, res.greeks[name], fd)


@pytest.mark.parametrize("paths", [1, 31, 129])
def test_few_paths_give_the_greeks_of_those_paths(paths):
    """No in-the-money path is lost or counted twice: a put so deep in the
    money that every path pays has delta -e^(-rT) mean(S_T) / S0, and
    mean(S_T) is K - price e^(rT)."""
    spec = HestonAdjointSpec(strike=1000.0, expiry=1.0, num_paths=paths, num_steps=8, seed=5, asian=False,
                             option_type=OptionType.Put)
    res = heston_adjoint(spec, **BASE)
    df = math.exp(-0.03)
    assert res.greeks["spot"] == pytest.approx(-(1000.0 * df - res.price) / 100.0, rel=1e-5)


@pytest.mark.parametrize("asian", [False, True])
def test_both_passes_give_the_same_greeks(asian):
    """Strikes 1e-6 apart on the two sides of the rule: the same paths, 1e-5 of
    whose in-the-money ones change sides.  Either pass is within 1e-3 (2e-4
    absolute) of the FP64 difference, so within twice that of the other."""
    T, mu = 1.0, BASE["rate"]
    w = BASE["theta"] * T / (3.0 if asian else 1.0)
    f = math.log(math.expm1(mu * T) / (mu * T)) if asian else mu * T
    lo, hi = 0.0, 5.0  # d with normal cdf(-d) = 0.1
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if 0.5 * math.erfc(mid / math.sqrt(2.0)) > 0.1 else (lo, mid)
    K = 100.0 * math.exp(f - 0.5 * w + lo * math.sqrt(w))
    got = [heston_adjoint(HestonAdjointSpec(strike=K * x, expiry=T, num_paths=1 << 20, num_steps=65, seed=3,
                                            asian=asian), **BASE) for x in (1.0 - 5e-7, 1.0 + 5e-7)]
    assert got[0].price == pytest.approx(got[1].price, rel=1e-4)
    for name in A.OF_ADJ_NAMES:
        a, b = got[0].greeks[name], got[1].greeks[name]
        assert abs(a - b) <= 2.0 * max(1e-3 * abs(b), 2e-4), (name, a, b)


def test_the_longest_path_and_past_it():
    """2,048 steps fill the table of counter terms; one more is refused."""
    from openferric_b200 import PricingError
    spec = HestonAdjointSpec(strike=100.0, expiry=1.0, num_paths=4097, num_steps=2048, seed=5, asian=True)
    res = heston_adjoint(spec, **BASE)
    assert res.price == heston_adjoint(spec, forward_only=1, **BASE).price
    assert abs(res.price - heston_adjoint(spec, forward_only=2, **BASE).price) <= 1e-4 * res.price
    with pytest.raises(PricingError):
        heston_adjoint(HestonAdjointSpec(strike=100.0, expiry=1.0, num_paths=64, num_steps=2049, seed=5), **BASE)
