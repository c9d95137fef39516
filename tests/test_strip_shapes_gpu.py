"""The strip's tile shapes (one sample per thread, two in packed pairs, producer
and consumer warps) round a path alike: with one sample there is one path and
one payoff, so prices are equal in every bit, whatever the step count leaves of
the last counter block.  In the money at any draw, so that no shape prices 0."""
import pytest

import openferric_b200 as of
from openferric_b200 import OptionType
from openferric_b200.engines import price_strike_strip

pytestmark = pytest.mark.gpu


def _gen(model, steps):
    if model == "gbm":
        return of.GbmPathGenerator(of.Gbm(0.03, 0.25), 100.0, 1.0, steps)
    return of.HestonPathGenerator(of.Heston(0.03, 2.0, 0.04, 0.5, -0.7, 0.04), 100.0, 1.0, steps, model)


@pytest.mark.parametrize("model", ["gbm", "euler", "qe"])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 6, 7, 8, 63, 64, 65, 1027])
@pytest.mark.parametrize("anti", [False, True])
def test_one_path_is_the_same_in_every_shape(model, steps, anti):
    for seed in range(40):
        for strikes in ([1.0], [1.0, 2.0]):
            one, two, ws = (price_strike_strip(_gen(model, steps), OptionType.Call, strikes, 2 if anti else 1, seed,
                                               1.0, antithetic=anti, tile_ilp=tile) for tile in (1, 2, 3))
            assert one[0][0] > 1.0
            assert one == two, (seed, one, two)
            assert one == ws, (seed, one, ws)


@pytest.mark.parametrize("model", ["gbm", "euler", "qe"])
@pytest.mark.parametrize("tile", [1, 2])
def test_one_strike_pays_what_it_pays_beside_another(model, tile):
    for seed in range(100):
        alone, beside = (price_strike_strip(_gen(model, 5), OptionType.Call, strikes, 1, seed, 1.0, tile_ilp=tile)
                         for strikes in ([1.0], [1.0, 2.0]))
        assert alone[0] == beside[0], (seed, alone, beside)
