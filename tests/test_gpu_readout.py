"""hlbg_get_f on the host and on the device: every storage form, odd site counts, an
output that is only 8-byte aligned, and stored values of every kind (zeros, subnormal
deviations, infinities, NaN)."""
import numpy as np
import pytest

from hemelb_gb300 import capi, cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32DEV, capi.FP16])
@pytest.mark.parametrize("radius,length", [(4.0, 17), (6.0, 31)])
def test_read_of_the_distributions(prec, radius, length):
    c = cases.pipe(radius, length)
    s = c.solver(prec)
    rng = np.random.default_rng(1)
    g = 1e-3 * rng.standard_normal((s.n_sites, 19))
    for v in (0.0, -0.0, 1e-40, -1e-42, 5e-8, np.inf, -np.inf, np.nan):
        g[rng.integers(0, s.n_sites, 5), rng.integers(0, 19, 5)] = v
    f = g + W
    s.SetInitialConditions()
    s.PutF(f, 0)
    s.PutF(f, 1)
    if prec == capi.FP64:
        want = f
    elif prec == capi.FP32DEV:
        want = (f - W).astype(np.float32).astype(np.float64) + W
    else:
        with np.errstate(all="ignore"):
            want = ((f - W).astype(np.float32) * np.float32(1024)).astype(np.float16).astype(np.float32)
            want = (want * np.float32(1 / 1024)).astype(np.float64) + W
    assert np.array_equal(s.GetFOld(), want, equal_nan=True)
    assert np.array_equal(s.GetFNew(), want, equal_nan=True)
    for off in (0, 1):
        buf = torch.full((s.n_sites * 19 + 2,), -5.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        capi.check(capi.load().hlbg_get_f_device(s.ctx, buf.data_ptr() + 8 * off, 0), s.ctx)
        got = buf.cpu().numpy()
        assert np.array_equal(got[off:off + s.n_sites * 19].reshape(-1, 19), want, equal_nan=True)
        assert got[-1] == -5.0 and (off == 0 or got[0] == -5.0)
