"""The end of a training step as overlapped launches: Adam reads gradients that the kernels
before it add to, and the next forward pass reads the weights it writes."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn, surrogate  # noqa: E402
from tests.test_nn_launches_gpu import CALLS, _inputs  # noqa: E402

LR = 1e-3


def _grad(net, x, target, mask):
    out = net.forward(x)
    dout = torch.empty(out.shape, dtype=torch.bfloat16, device=out.device)
    nn.mse(out, target, mask, dout, torch.zeros(1, device=out.device))
    net.zero_grad()
    net.backward(dout)


def _net(scale):
    """Weights of seed 1 in mid-training: moments of the gradients' size, step 1,000."""
    net = surrogate.UNet(seed=1)
    net.t = 1000
    if scale is not None:
        g = torch.Generator(device="cuda").manual_seed(5)
        for c, (sw, sb) in zip(net.L.values(), scale):
            for m, v, s in ((c.mw, c.vw, sw), (c.mb, c.vb, sb)):
                m.copy_((2 * torch.rand(m.shape, generator=g, device="cuda") - 1) * s)
                v.fill_(s * s)
    return net


def _tensors(net):
    return [t for c in net.L.values() for t in ((c.w, c.gw), (c.b, c.gb))]


@pytest.mark.parametrize("b", [8, 24])
def test_update_and_the_pass_behind_it(b, monkeypatch):
    x, target, mask = _inputs(b)
    first = _net(None)
    _grad(first, x, target, mask)
    torch.cuda.synchronize()
    scale = [tuple(max(float(g.abs().max()), 1e-20) for g in (c.gw, c.gb)) for c in first.L.values()]

    def run(stream=None):
        nets = [_net(scale) for _ in range(3)]
        torch.cuda.synchronize()
        outs = []
        with torch.cuda.stream(stream):
            for net in nets:  # back to back
                _grad(net, x, target, mask)
                net.step(LR)
                outs.append(net.forward(x).clone())
        torch.cuda.synchronize()
        return nets, outs

    got = [run(), run(torch.cuda.Stream())]
    for name in CALLS:
        f = getattr(nn, name)

        def synced(*a, _f=f, **k):
            torch.cuda.synchronize()
            r = _f(*a, **k)
            torch.cuda.synchronize()
            return r
        monkeypatch.setattr(nn, name, synced)
    want = run()[0][0]
    scales = [s for pair in scale for s in pair]
    for nets, outs in got:
        for net, out in zip(nets, outs):
            # the pass behind the update read the whole of it
            assert torch.equal(out, net.forward(x))
            for c in net.L.values():
                assert torch.equal(c.wb, c.w.to(torch.bfloat16))
            for (w, g), (w0, g0), s in zip(_tensors(net), _tensors(want), scales):
                # FP32 sums in any order, as for the weight gradients of the launches' test
                tol = 2.0 ** -10 * float(g0.norm())
                assert float((g - g0).norm()) <= tol
                # |g| <= s, |m| <= s, v = s^2: an update changes by no more than lr (0.1 +
                # 0.016) / s times its gradient's change, and is rounded with its weight
                assert float((w - w0).norm()) <= LR * 0.116 / s * tol + 2.0 ** -22 * float(w0.norm()) + 1e-12
