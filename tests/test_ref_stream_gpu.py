"""The log-space kernels of the FP64 reference stream (mc_reference.cu) at
their edges: the last partial draw group and draw batch, partial warps and
blocks, grids that stride, every payoff they take.  A proportional dividend of
ratio 0 sends the same request through the general kernel, which multiplies
the spot step by step on the same draws.

Tolerance: the two sum or multiply at most 300 terms in another order, so S_T
agrees to 300 x 2^-53 = 3.3e-14 relative; a price here is more than 1/30 of
the spot whenever it is not 0, which gives 1e-12."""
import math

import numpy as np
import pytest

import openferric_b200 as of
from openferric_b200 import (AsianOption, AsianSpec, Averaging, BarrierOption, BarrierSpec, BarrierDirection,
                             BarrierStyle, ControlVariate, ControlVariateKind, DividendEvent, DividendSchedule,
                             FastRngKind, Gbm, GbmPathGenerator, MonteCarloEngine, OptionType, StrikeType,
                             VanillaOption)

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _asian(avg, strike_type, times, opt=OptionType.Call):
    return AsianOption(opt, 90.0, 1.0, AsianSpec(avg, strike_type, list(times)))


def _barrier(d, s, level, rebate=1.5):
    return BarrierOption(OptionType.Call, 90.0, 1.0, BarrierSpec(d, s, level, rebate))


def _instruments(steps):
    daily = [j / steps for j in range(1, steps + 1)]
    return {
        "call": VanillaOption.european_call(90.0, 1.0),
        "up_out": _barrier(BarrierDirection.Up, BarrierStyle.Out, 130.0),
        "down_in": _barrier(BarrierDirection.Down, BarrierStyle.In, 95.0),
        "at_spot": _barrier(BarrierDirection.Down, BarrierStyle.Out, 100.0),
        "arith": _asian(Averaging.Arithmetic, StrikeType.Fixed, daily),
        "arith_start": _asian(Averaging.Arithmetic, StrikeType.Fixed, [0.0, 0.31, 0.33, 1.0]),
        "geo": _asian(Averaging.Geometric, StrikeType.Fixed, daily),
        "floating": _asian(Averaging.Arithmetic, StrikeType.Floating, daily, OptionType.Put),
    }


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 15, 16, 17, 252])
@pytest.mark.parametrize("name", list(_instruments(1)))
@pytest.mark.parametrize("paths,anti,rng", [(1, False, "x"), (33, True, "x"), (64, False, "p"), (1001, True, "p"),
                                            (1001, False, "x")])
def test_log_space_kernels_match_the_general_kernel(steps, name, paths, anti, rng):
    inst = _instruments(steps)[name]
    noop = DividendSchedule.new([DividendEvent.proportional(0.5, 0.0)])
    res = []
    for div in (None, noop):
        eng = MonteCarloEngine(paths, 77).with_antithetic(anti) \
            .with_rng_kind(FastRngKind.Pcg64 if rng == "p" else FastRngKind.Xoshiro256PlusPlus)
        if name == "arith":
            eng.with_control_variate(ControlVariate(5.0, ControlVariateKind.GeometricAsian))
        res.append(eng.run_full(GbmPathGenerator(Gbm(0.03, 0.3), 100.0, 1.0, steps, div), inst, 0.97))
    fast, slow = res
    for f in ("sum_x", "sum_x2", "sum_y", "sum_xy", "sum_y2"):
        a, b = getattr(fast, f), getattr(slow, f)
        # a square or product has twice the relative error of a payoff; a payoff near 0 is bounded by the spot
        assert abs(a - b) <= 2 * RTOL * max(abs(b), paths * 100.0 ** (1 if f in ("sum_x", "sum_y") else 2) / 30), f


@pytest.mark.parametrize("name", ["call", "up_out", "arith"])
def test_more_samples_than_one_grid(name):
    """151,552 samples are 16 blocks of 64 on each of 148 SMs; more make the blocks stride."""
    inst = _instruments(3)[name]
    noop = DividendSchedule.new([DividendEvent.proportional(0.5, 0.0)])
    a, b = (MonteCarloEngine(200_001, 5).run_full(GbmPathGenerator(Gbm(0.03, 0.3), 100.0, 1.0, 3, d), inst, 0.97)
            for d in (None, noop))
    assert a.samples == b.samples == 200_001
    assert abs(a.price - b.price) <= RTOL * b.price and abs(a.stderr_ - b.stderr_) <= 1e-10 * b.stderr_


def test_wide_asian_takes_the_general_kernel():
    """A log-spot that could leave the table exponential's range: sigma sqrt(T) = 20."""
    inst = _asian(Averaging.Arithmetic, StrikeType.Fixed, [0.5, 1.0])
    noop = DividendSchedule.new([DividendEvent.proportional(0.5, 0.0)])
    a, b = (MonteCarloEngine(500, 5).run_full(GbmPathGenerator(Gbm(0.03, 20.0), 100.0, 1.0, 4, d), inst, 0.97)
            for d in (None, noop))
    assert a.price == b.price and math.isfinite(a.price)


@pytest.mark.parametrize("steps", [1, 7, 8, 9])
@pytest.mark.parametrize("anti", [False, True])
def test_heston_batches_match_the_injected_stream(orc, steps, anti):
    """The general kernel on the oracle's normals of the same stream, zero initial variance included."""
    for v0 in (0.04, 0.0):
        gen = of.HestonPathGenerator(of.Heston(0.03, 2.0, 0.04, 0.9, -0.7, v0), 100.0, 1.0, steps)
        inst = VanillaOption.european_call(90.0, 1.0)
        paths = 333
        z = orc.run_normals(11, (paths + 1) // 2 if anti else paths, steps, 2)
        own = MonteCarloEngine(paths, 11).with_antithetic(anti).run_full(gen, inst, 0.97)
        inj = MonteCarloEngine(paths, 11).with_antithetic(anti).with_injected_normals(np.asarray(z)).run_full(
            gen, inst, 0.97)
        assert abs(own.price - inj.price) <= RTOL * inj.price
        assert abs(own.stderr_ - inj.stderr_) <= 1e-10 * inj.stderr_
