"""of_min_sum_in_order (host code of the library) against the double loop it
restates: whole rows are added at a time only where that is the same sum bit
for bit, so schedules with rounding ties, crossings of a binade, zeros,
duplicates, no order, or values outside [0, 1e100] must all agree exactly."""
import math
import random
from array import array

import numpy as np
import pytest

from openferric_b200.analytic import fixing_array, min_sum_in_order


def _loop(t):
    s = 0.0
    for ti in t:
        for tj in t:
            s += tj if tj < ti else ti
    return s


def _schedules():
    rng = random.Random(5)
    yield "dyadic", [j / 64.0 for j in range(1, 321)]
    yield "ties at every binade", [(1 + j) * (1.0 + 2.0 ** -52) for j in range(200)]
    yield "daily", [5.0 * j / 1260 for j in range(1, 901)]
    yield "with zero", [j / 100.0 for j in range(0, 301)]
    yield "duplicates", [rng.choice([0.25, 0.3, 0.7]) for _ in range(300)]
    yield "unsorted", [rng.uniform(0.0, 30.0) for _ in range(400)]
    yield "wide", [10.0 ** rng.uniform(-12.0, 12.0) for _ in range(300)]
    yield "one large", [1e-3] * 200 + [1e9]
    yield "negative", [-1.0, 0.5, 2.0, -0.25] * 20
    yield "infinite", [1.0, math.inf, 2.0] * 10
    yield "huge", [1e120 * rng.random() for _ in range(50)]
    yield "subnormal", [5e-324 * k for k in range(60)]


@pytest.mark.parametrize("name,times", list(_schedules()), ids=[n for n, _ in _schedules()])
def test_row_sums_equal_the_double_loop(name, times):
    assert min_sum_in_order(times) == _loop(times)


def test_nan_stays_nan():
    assert math.isnan(min_sum_in_order([0.5, math.nan, 1.0]))


def test_fixing_array_takes_what_numpy_takes():
    for times in ([0.5, 1, np.float64(2.0)], (0.25, 0.5), np.arange(4.0)[::2], array("d", [1.0]), ["0.5", "1.5"], []):
        want = np.ascontiguousarray(times, dtype=np.float64)
        got = fixing_array(times)
        assert got.dtype == np.float64 and got.flags.c_contiguous and got.shape == want.shape and (got == want).all()
