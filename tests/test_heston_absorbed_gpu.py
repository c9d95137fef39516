"""Heston under theta = 0 in FP64: a variance that reaches 0 stays there
(v' = (1 - kappa dt) v + xi sqrt(v dt) z has no other source), in the log-space
kernels of the European price, of the delta and of the Longstaff-Schwartz
generator as in the general kernel and the oracle.

Tolerances as for theta > 0: the log-space step rounds a few times more, which
moves a path by 1e-15 relative.  A root near 0 magnifies that by 1/(2 sqrt(v)),
at most 1e3 over the 10^6 steps here (the smallest of them leaves v near 1e-7),
and the relative error of v halves with every root: below 1e-12 of a price."""
import math

import numpy as np
import pytest

import openferric_b200 as of
from openferric_b200 import Heston, MonteCarloEngine, OptionType, VanillaOption
from openferric_b200.greeks import HestonAadConfig, heston_price_delta_aad
from openferric_b200.lsm import LongstaffSchwartzEngine

pytestmark = pytest.mark.gpu

RTOL = 1e-12


@pytest.mark.parametrize("v0,xi,steps", [(0.0, 0.6, 256), (0.01, 0.5, 256), (0.01, 2.0, 50), (0.04, 0.9, 17)])
@pytest.mark.parametrize("anti", [False, True])
def test_european_matches_the_general_kernel(orc, v0, xi, steps, anti):
    gen = of.HestonPathGenerator(Heston(0.03, 2.0, 0.0, xi, -0.7, v0), 100.0, 1.0, steps)
    inst = VanillaOption(OptionType.Put, 104.0, 1.0)
    paths = 2001
    z = orc.run_normals(11, (paths + 1) // 2 if anti else paths, steps, 2)
    own, inj = (MonteCarloEngine(paths, 11).with_antithetic(anti).with_injected_normals(normals)
                .run_full(gen, inst, 0.97) for normals in (None, np.asarray(z)))
    assert inj.price > 0.0
    assert abs(own.price - inj.price) <= RTOL * inj.price
    if v0 > 0.0:
        assert abs(own.stderr_ - inj.stderr_) <= 1e-10 * inj.stderr_


def test_zero_variance_is_the_forward():
    """v0 = theta = 0: every path is the forward, whatever the draws."""
    gen = of.HestonPathGenerator(Heston(0.03, 2.0, 0.0, 0.6, -0.7, 0.0), 100.0, 1.0, 256)
    fwd = 100.0 * math.exp(0.03)
    r = MonteCarloEngine(100_000, 7).run_full(gen, VanillaOption.european_call(100.0, 1.0), 1.0)
    assert abs(r.price - (fwd - 100.0)) <= RTOL * fwd
    assert MonteCarloEngine(100_000, 7).run_full(gen, VanillaOption(OptionType.Put, 100.0, 1.0), 1.0).price == 0.0


@pytest.mark.parametrize("v0,xi,steps", [(0.0, 0.6, 256), (0.01, 0.5, 256), (0.01, 2.0, 50)])
def test_delta_matches_the_oracle(orc, v0, xi, steps):
    price, delta = heston_price_delta_aad(OptionType.Call, 101.0, 1.0, 100.0, 0.03,
                                          Heston(0.03, 2.0, 0.0, xi, -0.7, v0), HestonAadConfig(5000, steps, 7))
    p, d = orc.heston_price_delta(0, 101.0, 1.0, 100.0, 0.03, 0.03, 2.0, 0.0, xi, -0.7, v0, 5000, steps, 7)
    assert abs(price - p) <= RTOL * p and abs(delta - d) <= RTOL * d


@pytest.mark.parametrize("v0,xi,steps", [(0.01, 0.5, 100), (0.01, 2.0, 50), (0.04, 0.9, 20)])
def test_bermudan_matches_the_oracle(orc, v0, xi, steps):
    """Fitted values carry the conditioning of the normal equations, at most
    1e5 of a path's 1e-14: prices to 1e-9, the exercise counts exactly."""
    inst = of.BermudanOption.with_constant_strike(OptionType.Put, 103.0, 1.0, [0.2, 0.4, 0.6, 0.8, 1.0])
    m = of.Market.builder().spot(100.0).rate(0.02).dividend_yield(0.01).flat_vol(0.2).build()
    out = LongstaffSchwartzEngine(4001, steps, 321).with_heston_dynamics(Heston(0.0, 2.0, 0.0, xi, -0.5, v0)) \
        .price_bermudan_with_boundary(inst, m)
    p, se, recs = orc.lsm_bermudan(1, 1.0, inst.effective_schedule(), 100.0, 0.02, 0.01, 4001, steps, 321,
                                   dynamics=2, heston=(2.0, 0.0, xi, -0.5, v0))
    assert abs(out.result.price - p) <= 1e-9 * p
    assert [(b.itm_paths, b.exercised_paths) for b in out.exercise_boundary] == [(r[3], r[4]) for r in recs]
