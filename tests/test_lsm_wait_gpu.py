"""The wait of the FP64 backward induction's blocks for one another
(lsm_backward_ref, through of_test_lsm_wait): with every row it prices the put;
with one block's rows withheld every block gives up after the limit, the call
ends in a timeout and the context goes on pricing.  No GPU fault or hang is
involved: the failing wait is a loop on the global timer that ends by itself."""
import ctypes as C

import pytest

from openferric_b200 import Market, PricingError, VanillaOption
from openferric_b200._lib import context
from openferric_b200.lsm import LongstaffSchwartzEngine

pytestmark = pytest.mark.gpu


def _wait(withhold, limit_us):
    ctx, ok, us = context(0), C.c_int32(-1), C.c_double(-1.0)
    with ctx.lock:
        ctx.check(ctx._L.of_test_lsm_wait(ctx.handle, withhold, limit_us, C.byref(ok), C.byref(us)))
    return ok.value, us.value


def test_rows_that_arrive_are_seen():
    assert _wait(0, 500_000)[0] == 1


def test_a_withheld_row_ends_the_wait_and_the_context_survives():
    mk = Market.builder().spot(38.0).rate(0.05).flat_vol(0.3).build()
    put = VanillaOption.american_put(40.0, 1.0)
    before = LongstaffSchwartzEngine(1024, 4, 7).price(put, mk)
    assert _wait(0, 500_000)[0] == 1
    ok, us = _wait(1, 2000)
    assert ok == 0
    assert 2000.0 <= us < 500_000.0
    after = LongstaffSchwartzEngine(1024, 4, 7).price(put, mk)
    assert (after.price, after.stderr) == (before.price, before.stderr)
    assert _wait(0, 500_000)[0] == 1


def test_bad_limits_are_refused():
    with pytest.raises(PricingError, match="limit_us"):
        _wait(1, 0)
