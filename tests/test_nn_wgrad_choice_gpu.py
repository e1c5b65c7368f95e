"""Which kernel a weight gradient takes: on volumes a few voxels wide or high, mostly
padding of the tcgen05 kernel's 8 x 16 tiles, the other one, and the right sums from it."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import capi, nn  # noqa: E402


def _time(f, reps=20):
    best = 1e9
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(reps):
            f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best / reps


def _reference(x, dy, taps):
    d, h, w = x.shape[1:4]
    if taps == 1:
        return torch.einsum("ndhwo,ndhwi->oi", dy.double(), x.double())[None]
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    return torch.stack([torch.einsum("ndhwo,ndhwi->oi", dy.double(), xp[:, z:z + d, y:y + h, k:k + w])
                        for z in range(3) for y in range(3) for k in range(3)])


# us with mma.sync and with tcgen05 where they were measured apart
@pytest.mark.parametrize("cin,cout,vol,taps,thin", [
    (144, 48, (1, 96, 3, 3), 27, True),    # 13.1 and 29.7
    (288, 48, (3, 43, 4, 3), 27, True),    # 28.5 and 68.4
    (192, 32, (2, 22, 1, 48), 27, True),   # 29.5 and 65.5
    (48, 48, (1, 24, 24, 24), 27, False),  # 20.2 and 14.0
    (16, 48, (1, 3, 3, 3), 27, False),
    (192, 96, (1, 2, 2, 2), 1, False),
    (32, 16, (1, 4, 4, 1), 1, False),
    (32, 16, (1, 17, 1, 1), 1, False)])
def test_weight_gradient_takes_the_faster_kernel(cin, cout, vol, taps, thin):
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn((*vol, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn((*vol, cout), generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.zeros((taps, cout, cin), device="cuda")
    nn.conv3d_weight_grad(x, dy, dw)
    want = _reference(x, dy, taps)
    # FP32 sums of up to m products: m roundings of 2^-24 of the sum of magnitudes, taken
    # as at most sqrt(m) times the sum's norm
    m = x.numel() // cin
    assert float((dw - want).norm()) <= 2.0 ** -24 * m ** 1.5 * float(want.norm()) + 1e-6 * float(want.norm())
    if thin:
        lib = capi.load()
        tc = _time(lambda: lib.hlbg_nn_conv3d_wgrad_tc(x.data_ptr(), cin, dy.data_ptr(), cout, dw.data_ptr(), *vol, taps,
                                                       nn._stream()))
        # both sides measured beside the cases: the choice takes half the time; three
        # quarters leaves as much room to either side
        assert _time(lambda: nn.conv3d_weight_grad(x, dy, dw)) < 0.75 * tc
