"""The first replay of a strip plan that is created and launched while the
legacy default stream is busy: its ticket is zeroed on a stream of its own, so
the sums are those of later replays and nothing waits for the legacy stream."""
import pytest

from openferric_b200 import Gbm, GbmPathGenerator, OptionType
from openferric_b200.engines import StripPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strikes,paths", [(1, 10_000), (41, 1 << 14)])
def test_first_replay_beside_a_busy_legacy_stream(strikes, paths):
    import torch
    gen = GbmPathGenerator(Gbm(0.03, 0.25), 100.0, 1.0, 16)
    ks = [90.0 + k for k in range(strikes)]
    StripPlan(gen, OptionType.Call, ks, paths, 3, 0.97).close()  # kernels loaded
    busy = torch.zeros(1, device="cuda:0")
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the legacy stream
    busy += 1
    plan = StripPlan(gen, OptionType.Call, ks, paths, 3, 0.97)
    plan.launch()
    first = plan.results()
    torch.cuda.synchronize()
    plan.launch()
    second = plan.results()
    plan.close()
    assert first == second and all(p > 0.0 and se > 0.0 for p, se in first)
