"""The FP64 stream's path kernels draw what a path has: one step of 4,000,000
paths takes well under the time of twelve steps, in the kernel's own time.  (A
whole batch of 16 draws for every path took the same for one step as for
twelve, and twice a general kernel's time for one step.)"""
import pytest

import openferric_b200 as of
from openferric_b200 import (BarrierDirection, BarrierOption, BarrierSpec, BarrierStyle, MonteCarloEngine, OptionType,
                             VanillaOption)

pytestmark = pytest.mark.gpu


def _kernel_ms(model, steps):
    if model == "gbm":
        gen = of.GbmPathGenerator(of.Gbm(0.03, 0.25), 100.0, 1.0, steps)
        inst = BarrierOption(OptionType.Call, 100.0, 1.0, BarrierSpec(BarrierDirection.Up, BarrierStyle.Out, 130.0, 0.0))
    else:
        gen = of.HestonPathGenerator(of.Heston(0.03, 2.0, 0.04, 0.5, -0.7, 0.04), 100.0, 1.0, steps)
        inst = VanillaOption.european_call(100.0, 1.0)
    return min(MonteCarloEngine(4_000_000, 3).run_full(gen, inst, 1.0).kernel_ms for _ in range(9))


@pytest.mark.parametrize("model,many", [("gbm", 12), ("heston", 8)])
def test_one_step_costs_less_than_a_batch(model, many):
    assert _kernel_ms(model, 1) < 0.75 * _kernel_ms(model, many)
