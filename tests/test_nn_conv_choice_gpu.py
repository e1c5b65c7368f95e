"""Which kernel a convolution takes on volumes that are mostly padding of the tcgen05
kernel's tiles: the faster one, and the same bits from either."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn  # noqa: E402
from tests.test_nn_wgrad_choice_gpu import _time  # noqa: E402


@pytest.mark.parametrize("cin,cout,vol,thin", [
    (16, 48, (1, 96, 3, 3), True),      # us, mma.sync and tcgen05: 4.5 and 5.6
    (16, 48, (1, 48, 1, 48), True),     # 6.1 and 8.0
    (16, 144, (4, 13, 1, 11), True),    # 5.7 and 7.6
    (16, 48, (1, 48, 48, 1), False),    # 7.7 and 6.0
    (16, 96, (4, 2, 2, 2), False),      # 4.7 and 4.4
    (48, 48, (1, 96, 3, 3), False)])    # 9.2 and 7.8
def test_convolution_takes_the_faster_kernel(cin, cout, vol, thin):
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn((*vol, cin), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((27, cout, cin), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(cout, generator=g, device="cuda")
    out = {e: torch.empty((*vol, cout), dtype=torch.bfloat16, device="cuda") for e in ("auto", "tc", "mma")}
    for e, y in out.items():
        nn.conv3d(x, w, b, y, None, 27, True, engine=e)
    assert torch.equal(out["auto"], out["mma"]) and torch.equal(out["tc"], out["mma"])
    assert nn.mostly_padding(cin, cout, *vol) == thin

    def replay(engine):  # device time, 50 in a graph
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(50):
                nn.conv3d(x, w, b, out[engine], None, 27, True, engine=engine)
        return _time(graph.replay, 3)

    # the other kernel takes 1.24 to 1.34 times as long where the volume is thin
    if thin:
        assert replay("auto") < 0.9 * replay("tc")
