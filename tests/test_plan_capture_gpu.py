"""Plans created while the caller captures the context's stream (relaxed mode,
the one that allows allocation): their tables are on the device when they are
returned, outside the caller's graph, and launches after the capture (a graph cannot be
launched inside one) give the results of a plan that was created before it."""
import gc
import warnings

import pytest

from openferric_b200 import Gbm, GbmPathGenerator, Market, OptionType, VanillaOption
from openferric_b200 import _abi as A
from openferric_b200._lib import context
from openferric_b200.book import BookEntry, BookPlan
from openferric_b200.engines import StripPlan, VarianceReduction

pytestmark = pytest.mark.gpu


def _plan(kind):
    if kind == "strip":
        gen = GbmPathGenerator(Gbm(0.03, 0.25), 100.0, 1.0, 16)
        return StripPlan(gen, OptionType.Call, [95.0, 100.0, 105.0], 10_000, 3, 0.97)
    mk = Market.builder().spot(100.0).rate(0.03).flat_vol(0.3).build()
    book = [BookEntry(VanillaOption.european_call(95.0 + k, 1.0), mk, 5000, 16, VarianceReduction.None_)
            for k in range(300)]
    return BookPlan(book, seed=5, mode=A.OF_BOOK_GREEKS if kind == "greeks" else A.OF_BOOK_PRICE)


def _prices(plan):
    return plan.results() if isinstance(plan, StripPlan) else [(r.price, r.stderr) for r in plan.results()]


@pytest.mark.parametrize("kind", ["strip", "book", "greeks"])
def test_plan_created_under_capture(kind):
    import torch
    ctx = context(0)
    plan = _plan(kind)
    plan.launch()
    want = _prices(plan)
    plan.close()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    gc.collect()  # nothing that frees device memory may run inside the capture
    ctx.set_stream(stream.cuda_stream)
    try:
        with warnings.catch_warnings():  # a plan adds nothing to the caller's graph, which torch reports
            warnings.simplefilter("ignore")
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
                plan = _plan(kind)
        for _ in range(2):
            plan.launch()
            assert _prices(plan) == want
        plan.close()
        del graph
    finally:
        ctx.set_stream(0)
