"""The tcgen05 convolution's tiles against the mma.sync kernel, bit for bit (both add
the products of a slice of 16 channels, dz, dy, dx in the same order): volumes around
the 8 x 16 x planes tile, columns that end inside a tile, one to eighteen channel
slices in rows of 32, 64 and 128 bytes, more than 256 output channels, outputs that are
only 16-byte aligned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn  # noqa: E402
from oracle import nn_oracle as O  # noqa: E402


def _operands(shape, cin, cout, taps):
    g = torch.Generator(device="cuda").manual_seed(cin * 1000 + cout)
    x = torch.randn(shape + (cin,), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((taps, cout, cin), generator=g, device="cuda") / (taps * cin) ** 0.5).to(torch.bfloat16)
    return x, w, torch.randn(cout, generator=g, device="cuda")


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 5, 17, 9), (1, 9, 16, 8), (1, 13, 33, 24), (3, 2, 1, 40),
                                   (1, 31, 15, 7)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 16), (48, 80), (64, 48), (96, 96), (144, 48), (16, 272),
                                      (96, 288), (288, 32), (80, 256)])
def test_same_bits_as_mma_sync(shape, cin, cout):
    x, w, b = _operands(shape, cin, cout, 27)
    got = torch.empty(shape + (cout,), dtype=torch.bfloat16, device="cuda")
    want = torch.empty_like(got)
    got32 = torch.empty(shape + (cout,), device="cuda")
    want32 = torch.empty_like(got32)
    nn.tc_error(reset=True)
    for bias, relu in ((b, True), (None, False)):
        nn.conv3d(x, w, bias, want, want32, relu=relu, engine="mma")
        nn.conv3d(x, w, bias, got, got32, relu=relu, engine="tc")
        assert torch.equal(got32, want32) and torch.equal(got, want)
    assert nn.tc_error() == 0


def test_whole_network_sizes_and_a_float64_reference():
    """A volume of many tiles per CTA (persistent CTAs, both sets of accumulators)."""
    shape, cin, cout = (2, 50, 52, 44), 16, 32
    x, w, b = _operands(shape, cin, cout, 27)
    got = torch.empty(shape + (cout,), dtype=torch.bfloat16, device="cuda")
    got32 = torch.empty(shape + (cout,), device="cuda")
    want, want32 = torch.empty_like(got), torch.empty_like(got32)
    nn.conv3d(x, w, b, want, want32, relu=True, engine="mma")
    nn.conv3d(x, w, b, got, got32, relu=True, engine="tc")
    assert torch.equal(got32, want32) and torch.equal(got, want)
    ref = O.conv3d(x[:, :6, :6, :6].double().cpu().numpy(), w.double().cpu().numpy(),
                   b.double().cpu().numpy(), relu=True)
    # interior of the sub-volume; FP32 accumulation of 432 exact products: 432 * 2^-24 of
    # the sum of magnitudes (each output is a sum of 432 terms of size about 1/21)
    assert np.abs(got32[:, 1:5, 1:5, 1:5].double().cpu().numpy() - ref[:, 1:5, 1:5, 1:5]).max() <= 1e-3


@pytest.mark.parametrize("off", [8, 16])
@pytest.mark.parametrize("taps", [1, 27])
def test_outputs_off_a_32_byte_boundary(taps, off):
    shape, cin, cout = (1, 4, 18, 10), 32, 48
    x, w, b = _operands(shape, cin, cout, taps)
    n = 4 * 18 * 10 * cout
    want = torch.empty(shape + (cout,), dtype=torch.bfloat16, device="cuda")
    want32 = torch.empty(shape + (cout,), device="cuda")
    nn.conv3d(x, w, b, want, want32, taps=taps, engine="mma")
    buf = torch.full((n + 32,), 7.0, dtype=torch.bfloat16, device="cuda")
    buf32 = torch.full((n + 32,), 7.0, device="cuda")
    got, got32 = buf[off:off + n].view(shape + (cout,)), buf32[off // 2:off // 2 + n].view(shape + (cout,))
    nn.conv3d(x, w, b, got, got32, taps=taps, engine="tc")
    assert torch.equal(got, want) and torch.equal(got32, want32)
    assert bool((buf[:off] == 7).all()) and bool((buf[off + n:] == 7).all())
    assert bool((buf32[:off // 2] == 7).all()) and bool((buf32[off // 2 + n:] == 7).all())


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 5, 17, 9), (1, 13, 33, 24), (3, 2, 1, 40)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (48, 80), (144, 48), (16, 272)])
def test_1x1x1_same_bits_as_mma_sync(shape, cin, cout):
    """Planes without a halo; one slice (planes in any order) and several."""
    x, w, b = _operands(shape, cin, cout, 1)
    got = torch.empty(shape + (cout,), dtype=torch.bfloat16, device="cuda")
    got32 = torch.empty(shape + (cout,), device="cuda")
    want, want32 = torch.empty_like(got), torch.empty_like(got32)
    nn.tc_error(reset=True)
    nn.conv3d(x, w, b, want, want32, taps=1, relu=True, engine="mma")
    nn.conv3d(x, w, b, got, got32, taps=1, relu=True, engine="tc")
    assert torch.equal(got32, want32) and torch.equal(got, want)
    assert nn.tc_error() == 0
