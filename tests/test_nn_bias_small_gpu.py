"""Bias gradients of small tensors, in the scalar and in the vector kernel: against 64
bits, and few channels in no more time than the scalar kernel takes."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn  # noqa: E402
from tests.test_nn_wgrad_choice_gpu import _time  # noqa: E402


@pytest.mark.parametrize("c", [8, 16, 24, 40, 72, 192, 1024, 2048])
@pytest.mark.parametrize("m", [1, 2, 7, 216, 1024, 1731, 2049])
def test_sums_of_every_row_count(c, m):
    g = torch.Generator(device="cuda").manual_seed(c + m)
    dy = torch.randn((m, c), generator=g, device="cuda").to(torch.bfloat16)
    y = torch.randn((m, c), generator=g, device="cuda").to(torch.bfloat16)
    db = torch.full((c,), 0.5, device="cuda")
    nn.bias_grad(dy, db)
    # m roundings of 2^-24 of the sum of magnitudes
    bound = (m + 2) * 2.0 ** -24 * (dy.double().abs().sum(0) + 0.5)
    assert ((db - dy.double().sum(0) - 0.5).abs() <= bound).all()
    want = torch.where(y > 0, dy, torch.zeros_like(dy))
    db.fill_(0.5)
    nn.relu_bias_backward(dy, y, db)
    assert torch.equal(dy, want)
    assert ((db - want.double().sum(0) - 0.5).abs() <= bound).all()


@pytest.mark.parametrize("m", [8, 216])
def test_eight_channels_take_no_longer_than_in_the_scalar_kernel(m):
    store = torch.randn(8 * m + 8, device="cuda").to(torch.bfloat16)
    db = torch.zeros(8, device="cuda")

    def replay(dy):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(100):
                nn.bias_grad(dy, db)
        return _time(graph.replay, 3)

    # an odd offset goes to the scalar kernel; 1.5 us there and 2.4 in the vector kernel,
    # 1.25 times is half way
    assert replay(store[: 8 * m].view(m, 8)) < 1.25 * replay(store[1: 8 * m + 1].view(m, 8))


@pytest.mark.parametrize("n", [1, 8, 262143, 262144, 262152])
def test_relu_mask_in_either_kernel(n):
    dy = torch.randn(n, device="cuda").to(torch.bfloat16)
    y = torch.randn(n, device="cuda").to(torch.bfloat16)
    y[::5] = 0.0
    y[3::7] = float("nan")
    want = torch.where(y > 0, dy, torch.zeros_like(dy))
    nn.relu_backward(dy, y)
    assert torch.equal(dy, want)


def test_small_relu_mask_takes_no_longer_than_in_the_scalar_kernel():
    """1.1 us there and 1.3 in the vector kernel (216 voxels of 144 channels); 10 % more is
    half way."""
    store = torch.randn((2, 31104 + 8), device="cuda").to(torch.bfloat16)

    def replay(k):  # an odd offset goes to the scalar kernel
        dy, y = store[0, k: 31104 + k], store[1, k: 31104 + k]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(200):
                nn.relu_backward(dy, y)
        return _time(graph.replay, 5)

    assert replay(0) < 1.1 * replay(1)
