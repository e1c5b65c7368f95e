"""Python side of the surrogate's kernels (include/hemelb_gb300_nn.h).

Each function takes torch CUDA tensors as plain device memory (channels-last
BF16 activations, [taps][C_out][C_in] BF16 weights, FP32 gradients and master
weights), checks shapes and dtypes, and enqueues the library's kernel on torch's
current stream.  There is no fallback: the kernels are the implementation.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import capi

_BF16 = torch.bfloat16
_F32 = torch.float32


def _lib():
    return capi.load()


def _stream():
    # torch.cuda.current_stream().cuda_stream without the Stream object (8 us a launch)
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _p(t):
    return t.data_ptr() if t is not None else None


def _need(t, dtype, what):
    if t.dtype != dtype or not t.is_cuda or not t.is_contiguous():
        raise ValueError(f"{what}: need a contiguous CUDA {dtype} tensor, got {t.dtype} "
                         f"{'cuda' if t.is_cuda else 'cpu'} contiguous={t.is_contiguous()}")


def _ok(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} failed with status {rc}")


def tc_eligible(cin: int, cout: int, *tensors) -> bool:
    """Shapes the tcgen05 convolution takes: C_in and C_out multiples of 16, 16-byte
    aligned buffers."""
    if cin % 16 or cout % 16 or cout < 16:
        return False
    for t in tensors:
        if t is not None and t.data_ptr() % 16:
            return False
    return True


def tc_tiles(n: int, d: int, h: int, w: int) -> int:
    """Tiles of 8 x 16 x 2 output voxels of a volume (ragged ones whole)."""
    return n * -(-d // 2) * -(-h // 16) * -(-w // 8)


def tc_faster(cin: int, cout: int, voxels: int, taps: int) -> bool:
    """Where the tcgen05 convolution is the faster one (the two give the same bits): all
    but small volumes at 16 -> 16 channels and of the 1x1x1 convolution, whose one slice
    the mma.sync kernel finishes in less than a tcgen05 CTA's set-up.  Measured, us,
    mma.sync / tcgen05: 16 -> 16 at 12^3 4.3 / 5.2, 24^3 6.0 / 6.5, 48^3 20.5 / 13.7;
    48 -> 48 at 8^3 9.4 / 9.1; 192 -> 192 at 6^3 61 / 27."""
    return voxels >= 1 << 15 or (taps == 27 and cin * cout > 256)


def mostly_padding(cin: int, cout: int, n: int, d: int, h: int, w: int) -> bool:
    """Volumes that fill less than a fifth of the tcgen05 convolution's 8 x 16 tiles and are
    more of them than of the mma.sync kernel's bricks of 4 x 4 x 8, where that one is the
    faster one: at 16 input channels (one slice of work a tile) and where it takes its 16
    output channels a CTA (C_out no multiple of 32).  16 -> 48, us, mma.sync / tcgen05:
    96 x 3 x 3 voxels 4.5 / 5.6, 48 x 1 x 48 6.1 / 8.0, 1 3.7 / 4.1, but 48 x 48 x 1 7.7 /
    6.0.  Elsewhere tcgen05 is faster, or at most 5 % slower, for all but 19 of 1,447
    shapes (31 % at worst)."""
    tiles = n * d * -(-h // 16) * -(-w // 8)
    bricks = n * -(-d // 4) * -(-h // 4) * -(-w // 8)
    return cin == 16 and cout % 32 != 0 and 5 * n * d * h * w < 128 * tiles and (tiles > bricks or tiles <= 2)


def conv3d(x, w, bias, out, out_f32=None, taps=27, relu=False, engine="auto"):
    """out[n,z,y,x,co] = act(sum_{tap,ci} x[n,(z,y,x)+off(tap),ci] w[tap,co,ci] + bias[co]).

    engine "tc": the tcgen05 / TMEM / TMA kernel (hlbg_nn_conv3d_tc); "mma": the
    mma.sync kernel (hlbg_nn_conv3d, every shape); "auto": tcgen05 where it takes
    the shape, else mma.sync."""
    _need(x, _BF16, "conv3d input")
    _need(w, _BF16, "conv3d weights")
    _need(out, _BF16, "conv3d output")
    n, d, h, wd, cin = x.shape
    t, cout, cin_w = w.shape
    if t != taps or cin_w != cin or out.shape != (n, d, h, wd, cout):
        raise ValueError(f"conv3d shapes: x {tuple(x.shape)} w {tuple(w.shape)} out {tuple(out.shape)}")
    if bias is not None:
        _need(bias, _F32, "conv3d bias")
    if out_f32 is not None:
        _need(out_f32, _F32, "conv3d FP32 output")
    if engine == "auto":
        engine = ("tc" if tc_eligible(cin, cout, x, w, out, out_f32) and tc_faster(cin, cout, n * d * h * wd, taps)
                  and not (taps == 27 and mostly_padding(cin, cout, n, d, h, wd)) else "mma")
    lib = _lib()
    fn = lib.hlbg_nn_conv3d_tc if engine == "tc" else lib.hlbg_nn_conv3d
    _ok(fn(_p(x), cin, _p(w), _p(bias), _p(out), _p(out_f32), cout, n, d, h, wd, taps, int(relu), _stream()),
        "hlbg_nn_conv3d_tc" if engine == "tc" else "hlbg_nn_conv3d")


def conv3d_tc(x, w, bias, out, out_f32=None, taps=27, relu=False):
    """conv3d on the tcgen05 tensor cores (cin and cout multiples of 16)."""
    conv3d(x, w, bias, out, out_f32, taps, relu, engine="tc")


def tc_error(reset: bool = True) -> int:
    """Nonzero when a bounded wait of a tcgen05 convolution gave up."""
    return int(_lib().hlbg_nn_tc_error(int(reset)))


def flip_transpose(w, wt):
    _need(w, _BF16, "weights")
    _need(wt, _BF16, "flipped weights")
    taps, cout, cin = w.shape
    if wt.shape != (taps, cin, cout):
        raise ValueError("flip_transpose shapes")
    _ok(_lib().hlbg_nn_flip_transpose(_p(w), _p(wt), cout, cin, taps, _stream()), "hlbg_nn_flip_transpose")


def conv3d_data_grad(dy, w, dx, dx_f32=None, wt=None, engine="auto"):
    """dx = conv(dy, flipped transposed w): the input gradient of conv3d."""
    taps, cout, cin = w.shape
    if wt is None:
        wt = torch.empty((taps, cin, cout), dtype=_BF16, device=w.device)
    flip_transpose(w, wt)
    conv3d(dy, wt, None, dx, dx_f32, taps=taps, relu=False, engine=engine)


def conv3d_weight_grad(x, dy, dw):
    """dw[tap,co,ci] += sum over voxels of dy[m,co] x[m+off(tap),ci] (FP32 accumulate)."""
    _need(x, _BF16, "wgrad input")
    _need(dy, _BF16, "wgrad output gradient")
    _need(dw, _F32, "wgrad weight gradient")
    n, d, h, wd, cin = x.shape
    taps, cout, cin_w = dw.shape
    if cin_w != cin or dy.shape != (n, d, h, wd, cout):
        raise ValueError("conv3d_weight_grad shapes")
    _ok(_lib().hlbg_nn_conv3d_wgrad(_p(x), cin, _p(dy), cout, _p(dw), n, d, h, wd, taps, _stream()),
        "hlbg_nn_conv3d_wgrad")


def relu_backward(dy, y):
    _need(dy, _BF16, "relu dy")
    _need(y, _BF16, "relu y")
    _ok(_lib().hlbg_nn_relu_bwd(_p(dy), _p(y), dy.numel(), _stream()), "hlbg_nn_relu_bwd")


def bias_grad(dy, db):
    _need(dy, _BF16, "bias dy")
    _need(db, _F32, "bias gradient")
    c = dy.shape[-1]
    _ok(_lib().hlbg_nn_bias_grad(_p(dy), _p(db), dy.numel() // c, c, _stream()), "hlbg_nn_bias_grad")


def relu_bias_backward(dy, y, db):
    """relu_backward and bias_grad in one pass over dy."""
    _need(dy, _BF16, "relu dy")
    _need(y, _BF16, "relu y")
    _need(db, _F32, "bias gradient")
    c = dy.shape[-1]
    _ok(_lib().hlbg_nn_relu_bias_bwd(_p(dy), _p(y), _p(db), dy.numel() // c, c, _stream()), "hlbg_nn_relu_bias_bwd")


def pool2(x, y):
    _need(x, _BF16, "pool input")
    _need(y, _BF16, "pool output")
    n, d, h, w, c = x.shape
    _ok(_lib().hlbg_nn_pool2(_p(x), _p(y), n, d, h, w, c, 0, _stream()), "hlbg_nn_pool2")


def pool2_backward(dy, dx):
    n, d, h, w, c = dx.shape
    _need(dy, _BF16, "pool dy")
    _need(dx, _BF16, "pool dx")
    _ok(_lib().hlbg_nn_pool2(_p(dy), _p(dx), n, d, h, w, c, 1, _stream()), "hlbg_nn_pool2")


def _fused(c, d, h, w, *tensors):
    """Shapes the fused up/down-sampling passes take."""
    return (all(k % 8 == 0 for k in c) and d % 2 == h % 2 == w % 2 == 0
            and all(t.data_ptr() % 16 == 0 and 0 < t.numel() < 1 << 33 for t in tensors))


def pool2_backward_add(dy, acc):
    """acc += the gradient of pool2 (rounded to BF16, then added)."""
    n, d, h, w, c = acc.shape
    _need(dy, _BF16, "pool dy")
    _need(acc, _BF16, "pool sum")
    if not _fused((c,), d, h, w, dy, acc):
        tmp = torch.empty(acc.shape, dtype=_BF16, device=acc.device)
        pool2_backward(dy, tmp)
        add_(acc, tmp)
        return
    _ok(_lib().hlbg_nn_pool2_bwd_add(_p(dy), _p(acc), n, d, h, w, c, _stream()), "hlbg_nn_pool2_bwd_add")


def up2_concat(x, skip, y):
    """y = [up2(x) | skip] in one pass."""
    n, d, h, w, cb = skip.shape
    ca = x.shape[-1]
    for t, what in ((x, "upsample input"), (skip, "concat skip"), (y, "concat y")):
        _need(t, _BF16, what)
    if not _fused((ca, cb), d, h, w, x, skip, y):
        u = torch.empty((n, d, h, w, ca), dtype=_BF16, device=x.device)
        up2(x, u)
        concat(u, skip, y)
        return
    _ok(_lib().hlbg_nn_up2_concat(_p(x), ca, _p(skip), cb, _p(y), n, d, h, w, _stream()), "hlbg_nn_up2_concat")


def up2_split(dy, dx, dskip):
    """The gradient of up2_concat: dx = up2_backward of dy's first channels, dskip the rest."""
    n, d, h, w, cb = dskip.shape
    ca = dx.shape[-1]
    for t, what in ((dy, "split y"), (dx, "upsample dx"), (dskip, "split skip")):
        _need(t, _BF16, what)
    if not _fused((ca, cb), d, h, w, dy, dx, dskip):
        g = torch.empty((n, d, h, w, ca), dtype=_BF16, device=dy.device)
        split(dy, g, dskip)
        up2_backward(g, dx)
        return
    _ok(_lib().hlbg_nn_up2_split(_p(dy), _p(dx), ca, _p(dskip), cb, n, d, h, w, _stream()), "hlbg_nn_up2_split")


def up2(x, y):
    _need(x, _BF16, "upsample input")
    _need(y, _BF16, "upsample output")
    n, d, h, w, c = y.shape
    _ok(_lib().hlbg_nn_up2(_p(x), _p(y), n, d, h, w, c, 0, _stream()), "hlbg_nn_up2")


def up2_backward(dy, dx):
    n, d, h, w, c = dx.shape
    _need(dy, _BF16, "upsample dy")
    _need(dx, _BF16, "upsample dx")
    _ok(_lib().hlbg_nn_up2(_p(dy), _p(dx), n, d, h, w, c, 1, _stream()), "hlbg_nn_up2")


def concat(a, b, y):
    ca, cb = a.shape[-1], b.shape[-1]
    m = a.numel() // ca
    for t, w in ((a, "concat a"), (b, "concat b"), (y, "concat y")):
        _need(t, _BF16, w)
    _ok(_lib().hlbg_nn_concat(_p(a), ca, _p(b), cb, _p(y), m, _stream()), "hlbg_nn_concat")


def split(y, da, db, accumulate_b=False):
    ca, cb = da.shape[-1], db.shape[-1]
    m = da.numel() // ca
    for t, w in ((y, "split y"), (da, "split da"), (db, "split db")):
        _need(t, _BF16, w)
    _ok(_lib().hlbg_nn_split(_p(y), _p(da), ca, _p(db), cb, m, int(accumulate_b), _stream()),
        "hlbg_nn_split")


def add_(a, b):
    _need(a, _BF16, "add a")
    _need(b, _BF16, "add b")
    _ok(_lib().hlbg_nn_add(_p(a), _p(b), a.numel(), _stream()), "hlbg_nn_add")


def mse(pred, target, mask, dpred, loss=None):
    """Masked mean squared error over voxels with mask 1; writes dpred and returns the
    loss (a host float when `loss` is None, else accumulated into the FP32 device scalar)."""
    _need(pred, _F32, "mse pred")
    _need(target, _F32, "mse target")
    _need(mask, _F32, "mse mask")
    _need(dpred, _BF16, "mse dpred")
    c = pred.shape[-1]
    m = pred.numel() // c
    cnt = float(mask.sum()) * c
    own = loss is None
    if own:
        loss = torch.zeros(1, dtype=_F32, device=pred.device)
    _ok(_lib().hlbg_nn_mse(_p(pred), _p(target), _p(mask), _p(dpred), _p(loss), m, c,
                           1.0 / max(cnt, 1.0), _stream()), "hlbg_nn_mse")
    return float(loss) / max(cnt, 1.0) if own else None


def adam(w, wb, g, m, v, lr, step, b1=0.9, b2=0.999, eps=1e-8):
    for t, n in ((w, "adam w"), (g, "adam g"), (m, "adam m"), (v, "adam v")):
        _need(t, _F32, n)
    if wb is not None:
        _need(wb, _BF16, "adam bf16 copy")
    _ok(_lib().hlbg_nn_adam(_p(w), _p(wb), _p(g), _p(m), _p(v), w.numel(), lr, b1, b2, eps, step,
                            _stream()), "hlbg_nn_adam")


def adam_list(tensors, lr, step, b1=0.9, b2=0.999, eps=1e-8):
    """adam for a list of (w, wb or None, g, m, v) in one launch per 32 tensors."""
    for w, wb, g, m, v in tensors:
        for t, n in ((w, "adam w"), (g, "adam g"), (m, "adam m"), (v, "adam v")):
            _need(t, _F32, n)
        if wb is not None:
            _need(wb, _BF16, "adam bf16 copy")
        if not w.numel() == g.numel() == m.numel() == v.numel() == (w if wb is None else wb).numel():
            raise ValueError("adam_list sizes")
    k = len(tensors)
    ptrs = [(C.c_void_p * k)(*map(_p, column)) for column in zip(*tensors)] if k else [None] * 5
    sizes = (C.c_int64 * k)(*(t[0].numel() for t in tensors))
    _ok(_lib().hlbg_nn_adam_list(*ptrs, sizes, k, lr, b1, b2, eps, step, _stream()), "hlbg_nn_adam_list")


def to_bf16(x, y):
    _need(x, _F32, "to_bf16 input")
    _need(y, _BF16, "to_bf16 output")
    _ok(_lib().hlbg_nn_to_bf16(_p(x), _p(y), x.numel(), _stream()), "hlbg_nn_to_bf16")
