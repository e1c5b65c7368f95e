"""The network's overlapped launches: each kernel starts beside the end of the one before
it, so a whole training step, with torch's own kernels in between, with reused buffers,
on a side stream and replayed as a graph, has to give what it gives with a
synchronisation after every call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn, surrogate  # noqa: E402

CALLS = ("conv3d", "up2_concat", "up2_split", "pool2", "pool2_backward_add", "flip_transpose", "adam_list",
         "relu_bias_backward", "bias_grad", "conv3d_weight_grad", "mse")


def _step(net, x, target, mask):
    out = net.forward(x)
    dout = torch.empty(out.shape, dtype=torch.bfloat16, device=out.device)
    loss = torch.zeros(1, device=out.device)
    nn.mse(out, target, mask, dout, loss)
    net.zero_grad()
    net.backward(dout)
    net.step(1e-3)
    return out


def _inputs(b):
    g = torch.Generator(device="cuda").manual_seed(b)
    x = torch.randn((2, b, b, b, 16), generator=g, device="cuda").to(torch.bfloat16)
    return x, torch.randn((2, b, b, b, 16), generator=g, device="cuda"), torch.ones((2, b, b, b), device="cuda")


@pytest.mark.parametrize("b", [8, 24])
def test_a_training_step_as_with_a_synchronisation_after_every_call(b, monkeypatch):
    """One step from the same weights (a second step starts from weights whose first Adam
    update has the sign of gradients that round to either side of zero)."""
    x, target, mask = _inputs(b)

    def run(stream=None):
        nets = [surrogate.UNet(seed=1) for _ in range(3)]
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            outs = [_step(net, x, target, mask) for net in nets]  # back to back
        torch.cuda.synchronize()
        return outs, [[c.gw for c in net.L.values()] for net in nets]

    got = [run(), run(torch.cuda.Stream())]
    for name in CALLS:
        f = getattr(nn, name)

        def synced(*a, _f=f, **k):
            torch.cuda.synchronize()
            r = _f(*a, **k)
            torch.cuda.synchronize()
            return r
        monkeypatch.setattr(nn, name, synced)
    want, gw_want = run()
    for outs, gw in got:
        for a, grads in zip(outs, gw):
            assert torch.equal(a, want[0])  # the forward pass has no sums in an open order
            # a weight gradient adds the FP32 sums of its runs of voxels (fewer than 2^10)
            # in any order: 2^10 additions of 2^-24 of the sum of magnitudes, taken as at
            # most 2^4 of the sum's norm
            for g, w in zip(grads, gw_want[0]):
                assert float((g - w).norm()) <= 2.0 ** -10 * float(w.norm())


def test_forward_pass_captured_as_a_graph():
    x = _inputs(16)[0]
    net = surrogate.UNet(seed=2)
    want = net.forward(x).clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = net.forward(x)
    x.mul_(2)
    want2 = net.forward(x).clone()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want2) and not np.array_equal(want.cpu().numpy(), want2.cpu().numpy())
