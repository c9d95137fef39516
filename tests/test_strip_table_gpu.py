"""The strip's paths across the end of its table of Philox terms (1,792 counter
blocks: 7,168 GBM or 3,584 Heston steps), past which the terms are computed in
place: prices on the strip's own draws, paths in numpy and FP64, with
the tolerance derived beside them."""
import numpy as np
import pytest

from openferric_b200 import OptionType
from openferric_b200.engines import price_strike_strip
from test_strip_draws_gpu import S0, _gen, _paths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,steps", [("gbm", 7167), ("gbm", 7168), ("gbm", 7172), ("gbm", 7177),
                                         ("heston", 3583), ("heston", 3584), ("heston", 3585), ("heston", 3589),
                                         ("qe", 3586)])
@pytest.mark.parametrize("anti", [False, True])
@pytest.mark.parametrize("tile", [1, 2])
def test_paths_across_the_end_of_the_table(model, steps, anti, tile):
    samples, ks = 65, [92.0, 104.0]
    got = price_strike_strip(_gen(model, steps), OptionType.Call, ks, 2 * samples if anti else samples, 9, 1.0,
                             antithetic=anti, tile_ilp=tile)
    ends = [_paths(model, steps, samples, 9, s) for s in ((1, -1) if anti else (1,))]
    tol = S0 * (steps * 2.0 ** -23 + 2e-5)
    for k, (p, _) in zip(ks, got):
        x = sum(np.maximum(s - k, 0.0) for s in ends) / len(ends)
        assert abs(p - x.mean()) <= tol, (k, p, x.mean())
