"""The C entry of_min_sum_in_order itself (analytic.min_sum_in_order falls back
to numpy without the library, so a test through it may run neither): bit for
bit the double loop it restates where rows are added at a time, where they tie,
cross a binade or are not plain, and an error status, not an exception, when
its tables cannot be allocated."""
import ctypes as C
import math
import os
import random
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from openferric_b200 import _abi as A
from openferric_b200 import _lib

pytestmark = pytest.mark.skipif(not os.path.exists(_lib.LIB_PATH), reason="needs the built library")


def _entry(times):
    t = np.ascontiguousarray(times, dtype=np.float64)
    out = C.c_double(-1.0)
    assert _lib.load().of_min_sum_in_order(t.ctypes.data, t.size, C.byref(out)) == A.OF_OK
    return out.value


def _loop(t):
    s = 0.0
    for ti in t:
        for tj in t:
            s += tj if tj < ti else ti
    return s


def _schedules():
    rng = random.Random(6)
    yield "none", []
    yield "one", [0.7]
    yield "dyadic", [j / 64.0 for j in range(1, 321)]
    yield "ties at every binade", [(1 + j) * (1.0 + 2.0 ** -52) for j in range(200)]
    yield "ties of half a grid step", [0.5 + 2.0 ** -k for k in range(30, 54)] * 12
    yield "daily", [5.0 * j / 1260 for j in range(1, 901)]
    yield "descending", [j / 252.0 for j in range(252, 0, -1)]
    yield "zeros", [0.0] * 50 + [1.0] * 3
    yield "wide", [10.0 ** rng.uniform(-12.0, 12.0) for _ in range(300)]
    yield "one large", [1e-3] * 200 + [1e9]
    yield "just plain", [1e100] * 20
    yield "not plain", [1.0, math.inf, 2.0, -1.0] * 10
    yield "tiny", [1e-205 * k for k in range(1, 60)]


@pytest.mark.parametrize("name,times", list(_schedules()), ids=[n for n, _ in _schedules()])
def test_entry_equals_the_double_loop(name, times):
    want, got = _loop(times), _entry(times)
    assert got == want or (math.isnan(got) and math.isnan(want))


def test_entry_refuses_bad_arguments():
    L, out, t = _lib.load(), C.c_double(), np.ones(2)
    assert L.of_min_sum_in_order(t.ctypes.data, -1, C.byref(out)) == A.OF_ERR_INVALID_INPUT
    assert L.of_min_sum_in_order(None, 2, C.byref(out)) == A.OF_ERR_INVALID_INPUT
    assert L.of_min_sum_in_order(t.ctypes.data, 2, None) == A.OF_ERR_INVALID_INPUT


@pytest.mark.parametrize("n", [1 << 50, 1 << 60])
def test_an_allocation_that_fails_is_a_status(n):
    """More than the address space, and more than a vector can name; nothing is
    read.  In a process of its own: an exception out of a C entry ends it."""
    code = ("import ctypes as C, numpy as np\nfrom openferric_b200 import _abi as A, _lib\n"
            "t, out = np.ones(2), C.c_double()\n"
            f"assert _lib.load().of_min_sum_in_order(t.ctypes.data, {n}, C.byref(out)) == A.OF_ERR_ALLOC\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
