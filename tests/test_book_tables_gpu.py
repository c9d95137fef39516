"""The book kernels' shared table of Philox terms (price and Greeks modes).

A launch whose options all fit the table (8,192 GBM steps, four to a counter
block) runs without a range test; one longer option sends the whole book to
the kernels that compute the terms past the table in place.  The streams are
numbered by position, so the other options of such a book must keep their
draws: they are the same FP32 arithmetic on the same normals, up to the
compiler's contraction, 1e-6 of the price as between tile shapes.  The long
option itself is checked against the closed form."""
import math

import pytest

from openferric_b200 import (AsianOption, AsianSpec, Averaging, BarrierDirection, BarrierOption, BarrierSpec,
                             BarrierStyle, Market, OptionType, StrikeType, VanillaOption, VarianceReduction)
from openferric_b200 import _abi as A
from openferric_b200.book import BookEntry, BookPlan, price_book, price_book_greeks

pytestmark = pytest.mark.gpu


def _book(steps, paths):
    mk = Market.builder().spot(100.0).rate(0.03).dividend_yield(0.01).flat_vol(0.3).build()
    obs = [j / steps for j in range(1, steps + 1)]
    insts = [VanillaOption.european_call(105.0, 1.0),
             AsianOption(OptionType.Call, 100.0, 1.0, AsianSpec(Averaging.Arithmetic, StrikeType.Fixed, obs)),
             BarrierOption(OptionType.Call, 100.0, 1.0, BarrierSpec(BarrierDirection.Up, BarrierStyle.Out, 140.0, 0.0)),
             BarrierOption(OptionType.Put, 100.0, 1.0, BarrierSpec(BarrierDirection.Down, BarrierStyle.In, 85.0, 0.0))]
    vrs = [VarianceReduction.None_, VarianceReduction.Antithetic]
    return mk, [BookEntry(i, mk, paths, steps, vr) for i in insts for vr in vrs]


@pytest.mark.parametrize("price", [price_book, price_book_greeks])
@pytest.mark.parametrize("steps", [1, 3, 4, 5, 63, 8190, 8192])
def test_a_book_keeps_its_draws_beside_a_longer_option(price, steps):
    mk, book = _book(steps, 1500)
    long = BookEntry(VanillaOption.european_call(100.0, 1.0), mk, 1 << 14, 8197, VarianceReduction.None_)
    alone, beside = ([getattr(r, "result", r) for r in price(b, seed=17)] for b in (book, book + [long]))
    for a, b in zip(alone, beside):
        assert abs(a.price - b.price) <= 1e-6 * abs(a.price) + 1e-9
        assert abs(a.stderr - b.stderr) <= 1e-5 * abs(a.stderr) + 1e-9
    d1 = (math.log(1.0) + 0.02 + 0.045) / 0.3
    cdf = lambda x: 0.5 * math.erfc(-x / math.sqrt(2.0))  # noqa: E731
    bs = 100.0 * math.exp(-0.01) * cdf(d1) - 100.0 * math.exp(-0.03) * cdf(d1 - 0.3)
    last = beside[-1]
    assert abs(last.price - bs) <= 4.5 * last.stderr


@pytest.mark.parametrize("greeks", [False, True])
@pytest.mark.parametrize("paths", [1, 31, 1 << 13, 9_000_000])
def test_a_call_and_a_plan_give_the_same_results(greeks, paths):
    """The call stages its tables in pinned memory up to 8 MB (262,144 tiles;
    9,000,000 samples in tiles of 32 are past it), the plan uploads its own."""
    mk, book = _book(1, paths)
    book = book[:2] + _book(5, 100)[1]
    kw = dict(seed=23, block=32, paths_per_thread=1)
    plan = BookPlan(book, mode=A.OF_BOOK_GREEKS if greeks else A.OF_BOOK_PRICE, **kw)
    for _ in range(2):  # the second launch finds its tile counters cleared
        plan.launch()
        want = plan.greeks_results() if greeks else plan.results()
    plan.close()
    got = price_book_greeks(book, **kw) if greeks else price_book(book, **kw)
    for g, w in zip(got, want):
        if greeks:
            assert (g.result.greeks, g.greeks_stderr) == (w.result.greeks, w.greeks_stderr)
            g, w = g.result, w.result
        assert (g.price, g.stderr) == (w.price, w.stderr)
