"""The FP64 Longstaff-Schwartz kernels at their edges.

The stream generator (a warp per 32, 64 or 128 paths, batches of 16 draws
that span paths) against the general generator fed with the oracle's normals
of the same stream; the one-launch backward induction against the launch per
date that a batch of many contracts takes.  Log-space paths differ from the
multiplied ones by a few 1e-15, fitted values by that times the conditioning
of the normal equations (at most 1e5 for the spots here), and no exercise
decision is that close: prices agree to 1e-9 with room, and to 1e-12 where
the spots are the same."""
import numpy as np
import pytest

import openferric_b200 as of
from openferric_b200 import Heston, OptionType, VanillaOption
from openferric_b200.lsm import LongstaffSchwartzEngine

pytestmark = pytest.mark.gpu


def _market():
    return of.Market.builder().spot(38.0).rate(0.05).dividend_yield(0.01).flat_vol(0.3).build()


@pytest.mark.parametrize("paths,steps", [(31, 2), (33, 15), (1024, 16), (1025, 17), (2500, 33), (59_999, 3),
                                         (60_001, 5), (149_999, 2), (150_001, 3)])
def test_stream_generator_matches_injected_normals(orc, paths, steps):
    z = np.asarray(orc.sequential_normals(9, paths * steps))
    opt = VanillaOption.american_put(40.0, 1.0)
    own = LongstaffSchwartzEngine(paths, steps, 9).price_with_delta(opt, _market())
    inj = LongstaffSchwartzEngine(paths, steps, 9).with_injected_normals(z).price_with_delta(opt, _market())
    assert abs(own.price - inj.price) <= 1e-9 * inj.price
    assert abs(own.stderr - inj.stderr) <= 1e-9 * inj.stderr
    assert abs(own.greeks.delta - inj.greeks.delta) <= 1e-9


@pytest.mark.parametrize("steps", [7, 8, 20])
@pytest.mark.parametrize("dynamics", ["heston", "local_vol"])
def test_two_draw_and_local_vol_streams(orc, steps, dynamics):
    paths, draws = 2001, 2 if dynamics == "heston" else 1
    inst = of.BermudanOption.with_constant_strike(OptionType.Put, 100.0, 1.0, [0.25, 0.5, 0.75, 1.0])
    m = of.Market.builder().spot(100).rate(0.02).vol_surface(lambda k, t: 0.2 + 0.1 * abs(k / 100.0 - 1.0)).build()
    z = np.asarray(orc.sequential_normals(4, paths * steps * draws))
    out = []
    for normals in (None, z):
        eng = LongstaffSchwartzEngine(paths, steps, 4).with_injected_normals(normals)
        eng = eng.with_heston_dynamics(Heston(0.0, 2.0, 0.04, 0.6, -0.5, 0.04)) if dynamics == "heston" \
            else eng.with_local_vol_dynamics()
        out.append(eng.price_bermudan_with_boundary(inst, m))
    own, inj = out
    assert abs(own.result.price - inj.result.price) <= 1e-9 * inj.result.price
    assert [(p.itm_paths, p.exercised_paths) for p in own.exercise_boundary] == \
        [(p.itm_paths, p.exercised_paths) for p in inj.exercise_boundary]


@pytest.mark.parametrize("degree", [2, 3])
@pytest.mark.parametrize("paths", [3, 255, 257, 1023, 4097, 20_000])
def test_one_launch_matches_a_launch_per_date(paths, degree):
    """200 contracts need more blocks than SMs, so the batch takes a launch per date."""
    eng = LongstaffSchwartzEngine(paths, 12, 3).with_basis_degree(degree)
    puts = [(VanillaOption.american_put(36.0 + 0.05 * k, 1.0), _market()) for k in range(200)]
    batch = eng.price_batch(puts, with_delta=True)
    for k in (0, 77, 199):
        one = eng.price_batch([puts[k]], with_delta=True)[0]
        assert abs(one.price - batch[k].price) <= 1e-12 * max(batch[k].price, 1.0)
        assert abs(one.greeks.delta - batch[k].greeks.delta) <= 1e-11


@pytest.mark.parametrize("paths", [37_000, 75_777, 151_000, 303_000, 606_000, 607_000])
def test_paths_per_thread_of_the_one_launch_induction(orc, paths):
    """1, 2, 4, 8 and 16 paths per thread on 148 SMs, and past them."""
    p, s = orc.lsm_price(1, 40.0, 1.0, 1, 38.0, 0.05, 0.01, 0.3, paths, 4, 21)
    r = LongstaffSchwartzEngine(paths, 4, 21).price(VanillaOption.american_put(40.0, 1.0), _market())
    assert abs(r.price - p) <= 1e-12 * p and abs(r.stderr - s) <= 1e-10 * s


def test_vol_beyond_the_table_exponential(orc):
    """sigma sqrt(T) = 20 takes the general generator."""
    m = of.Market.builder().spot(38.0).rate(0.05).flat_vol(20.0).build()
    r = LongstaffSchwartzEngine(2000, 6, 21).price(VanillaOption.american_put(40.0, 1.0), m)
    p, _ = orc.lsm_price(1, 40.0, 1.0, 1, 38.0, 0.05, 0.0, 20.0, 2000, 6, 21)
    assert abs(r.price - p) <= 1e-9 * p
