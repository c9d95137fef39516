"""Pinned staging of a Longstaff-Schwartz call with far more tables than the
context keeps a buffer for: 64 contracts of 32,767 dates need 128 MB on the host
and as much on the device.  The call gives the host's back, so the process's
address space, which holds both, grows by the device's alone; a call with as
large a path store and few dates goes first, so that everything else is there."""
import pytest

from openferric_b200 import Market, Precision, VanillaOption
from openferric_b200.lsm import LongstaffSchwartzEngine

pytestmark = pytest.mark.gpu


def _address_space_mb():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("VmSize:")) / 1024.0


def test_large_staging_is_given_back():
    mk = Market.builder().spot(38.0).rate(0.05).flat_vol(0.3).build()
    puts = [(VanillaOption.american_put(30.0 + 0.25 * k, 1.0), mk) for k in range(64)]

    def price(paths, steps):
        return LongstaffSchwartzEngine(paths, steps, 7).with_precision(Precision.Fp32Philox).price_batch(puts)

    price(600_000, 64)
    before = _address_space_mb()
    long = price(100, 32767)
    grown = _address_space_mb() - before
    short = price(100, 512)
    assert all(abs(a.price - b.price) < 6.0 * (a.stderr + b.stderr) + 0.2 for a, b in zip(long, short))
    assert grown < 192.0, grown
