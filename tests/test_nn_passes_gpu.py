"""The channels-last element-wise passes of the surrogate at the sizes where their
vector forms can go wrong: one group of 8 channels and many, row counts around the
CTA's, sizes the vector forms leave to the scalar ones (odd volumes, channel counts
that are no multiple of 8, buffers off a 16-byte boundary)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn  # noqa: E402

BF16 = torch.bfloat16


def _rand(shape, seed, off=0):
    """BF16 normal values; with `off`, in a buffer that starts off a 16-byte boundary."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = 1
    for k in shape:
        n *= k
    return torch.randn(n + off, generator=g, device="cuda").to(BF16)[off:].view(shape)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("m,c", [(1, 8), (5, 16), (127, 16), (513, 16), (4099, 48), (700, 192), (33, 24), (40, 12),
                                 (9, 2048), (70001, 16)])
def test_relu_and_bias_gradient(m, c, off):
    dy, y = _rand((m, c), 1, off), _rand((m, c), 2, off)
    y[0, 0] = float("nan")
    y[-1, -1] = 0.0
    want = torch.where(y > 0, dy, torch.zeros_like(dy))
    db = torch.full((c,), 0.5, device="cuda")
    alone, db1 = dy.clone(), torch.full((c,), 0.5, device="cuda")
    buf = torch.empty(m * c + off, dtype=BF16, device="cuda")[off:].view(m, c)
    buf.copy_(dy)
    nn.relu_bias_backward(buf, y, db)
    assert torch.equal(buf, want)
    buf.copy_(alone)
    nn.relu_backward(buf, y)
    assert torch.equal(buf, want)
    nn.bias_grad(buf, db1)
    ref = want.double().sum(0) + 0.5
    # FP32 sums of m terms of size 1 in blocks: well inside 1e-6 of sum |dy|
    tol = 1e-6 * (want.double().abs().sum(0) + 1)
    assert bool(((db.double() - ref).abs() <= tol).all()) and bool(((db1.double() - ref).abs() <= tol).all())


def _up(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)


def _sum8(g):
    """The 8 fine values of a coarse voxel added in z, y, x order, rounded once."""
    s = torch.zeros((g.shape[0],) + tuple(k // 2 for k in g.shape[1:4]) + (g.shape[-1],), device="cuda")
    for a in (0, 1):
        for b in (0, 1):
            for e in (0, 1):
                s += g[:, a::2, b::2, e::2].float()
    return s


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("shape,ca,cb", [((1, 2, 2, 2), 8, 8), ((2, 4, 6, 8), 16, 48), ((1, 10, 6, 14), 96, 24),
                                         ((3, 2, 8, 2), 12, 8)])
def test_resampling_passes(shape, ca, cb, off):
    n, d, h, w = shape
    coarse = (n, d // 2, h // 2, w // 2)
    x, skip, dy = _rand(coarse + (ca,), 3, off), _rand(shape + (cb,), 4, off), _rand(shape + (ca + cb,), 5, off)
    y = _rand(shape + (ca + cb,), 6, off)
    nn.up2_concat(x, skip, y)
    assert torch.equal(y, torch.cat([_up(x), skip], -1))
    dx, dskip = _rand(coarse + (ca,), 7, off), _rand(shape + (cb,), 8, off)
    nn.up2_split(dy, dx, dskip)
    assert torch.equal(dskip, dy[..., ca:]) and torch.equal(dx, _sum8(dy[..., :ca]).to(BF16))
    up = _rand(shape + (ca,), 9, off)
    nn.up2(x, up)
    assert torch.equal(up, _up(x))
    back = _rand(coarse + (ca,), 10, off)
    nn.up2_backward(up, back)
    assert torch.equal(back, _sum8(up).to(BF16))
    pooled = _rand(coarse + (ca,), 11, off)
    nn.pool2(up, pooled)
    assert torch.equal(pooled, (_sum8(up) * 0.125).to(BF16))
    grad = _rand(shape + (ca,), 12, off)
    acc = _rand(shape + (ca,), 13, off)
    want = (acc.float() + _up((x.float() * 0.125).to(BF16)).float()).to(BF16)
    nn.pool2_backward(x, grad)
    assert torch.equal(grad, _up((x.float() * 0.125).to(BF16)))
    nn.pool2_backward_add(x, acc)
    assert torch.equal(acc, want)


@pytest.mark.parametrize("m,c", [(1, 4), (255, 16), (70000, 16), (333, 12), (50, 5)])
def test_masked_loss(m, c):
    g = torch.Generator(device="cuda").manual_seed(m)
    p, t = torch.randn((m, c), generator=g, device="cuda"), torch.randn((m, c), generator=g, device="cuda")
    mask = (torch.rand(m, generator=g, device="cuda") > 0.4).float()
    mask[0] = 1.0
    d = torch.empty((m, c), dtype=BF16, device="cuda")
    loss = nn.mse(p, t, mask, d)
    diff = (p.double() - t.double()) * mask.double()[:, None]
    count = float(mask.sum()) * c
    assert abs(loss - float((diff ** 2).sum()) / count) <= 1e-6 * loss
    # FP32 difference and products (3 roundings of 2^-24), then one BF16 rounding
    assert bool(((d.double() - 2 * diff / count).abs() <= (2.0 ** -8) * (2 * diff / count).abs() + 1e-12).all())
