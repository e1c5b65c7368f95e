"""The tcgen05 weight gradient against the oracle: volumes around its 8 x 16 tile, every
row-group width of either operand (16, 32, 33-64, more than 64 channels), blocks that end
inside a group, both roles of x and dy, units that cross columns, 1x1x1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import capi, nn  # noqa: E402
from oracle import nn_oracle as O  # noqa: E402


def _tc(x, dy, dw):
    n, d, h, w, cin = x.shape
    taps, cout = dw.shape[:2]
    assert capi.load().hlbg_nn_conv3d_wgrad_tc(x.data_ptr(), cin, dy.data_ptr(), cout, dw.data_ptr(), n, d, h, w, taps,
                                               torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("taps", [27, 1])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (1, 3, 16, 8), (2, 5, 17, 9), (1, 2, 1, 25)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 16), (16, 48), (48, 32), (64, 64), (96, 16), (80, 96), (144, 48),
                                      (16, 272)])
def test_against_oracle(shape, cin, cout, taps):
    g = torch.Generator(device="cuda").manual_seed(cin + 7 * cout)
    x = torch.randn(shape + (cin,), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(shape + (cout,), generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.full((taps, cout, cin), 0.25, device="cuda")
    nn.tc_error(reset=True)
    _tc(x, dy, dw)
    assert nn.tc_error() == 0
    ref = O.conv3d_weight_grad(x.double().cpu().numpy(), dy.double().cpu().numpy(), taps=taps) + 0.25
    # FP32 sums of at most 2 * 5 * 17 * 9 products of size 1: well inside 1e-4 of the scale
    assert np.abs(dw.double().cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("cin,cout", [(16, 16), (64, 16), (48, 48)])
def test_long_sums_keep_fp32_accuracy(cin, cout):
    """Many units per CTA; the error against 64 bits is no larger than that of sums that
    are cut where the mma.sync kernel cuts them."""
    shape = (1, 40, 48, 40)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(shape + (cin,), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(shape + (cout,), generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.zeros((27, cout, cin), device="cuda")
    _tc(x, dy, dw)
    xd, gd = x.double(), dy.double()
    pad = torch.nn.functional.pad(xd, (0, 0, 1, 1, 1, 1, 1, 1))
    for tap in (0, 5, 13, 22, 26):
        dz, dyy, dx = tap // 9, tap // 3 % 3, tap % 3
        win = pad[:, dz:dz + 40, dyy:dyy + 48, dx:dx + 40].reshape(-1, cin)
        ref = gd.reshape(-1, cout).T @ win
        assert float((dw[tap].double() - ref).norm() / ref.norm()) <= 2e-6
