"""Readouts into host arrays of every kind: fresh pages, pages in use, an odd offset into
an allocation, pinned memory, on both sides of the size from which threads make the
pages present before the copy (4 MiB)."""
import ctypes as C

import numpy as np
import pytest
import torch

from hemelb_gb300 import capi, cases

pytestmark = pytest.mark.gpu


def _p(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _arrays(kind, n):
    if kind == "fresh":
        return np.empty(n)
    if kind == "used":
        return np.full(n, 7.0)
    if kind == "odd":  # 8 bytes past a page's start, guarded on both sides
        return np.full(n + 16, 7.0)[1: n + 1]
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("radius,length", [(8.0, 40.0), (22.0, 170.0)])  # u below, rho above 4 MiB
def test_readouts_are_the_same_in_every_kind_of_host_memory(radius, length):
    c = cases.bifurcation(seed=3, parent_radius=radius, parent_length=length, daughter_length_factor=2.0,
                          precision=capi.FP32DEV)
    s = c.solver()
    s.SetInitialConditions()
    s.DoTimeStep(2)
    n = s.n_sites
    assert (24 * n < 4 << 20) if radius < 10 else (8 * n >= 4 << 20)
    lib = capi.load()
    want = None
    for kind in ("used", "fresh", "odd", "pinned"):
        rho, u, f = _arrays(kind, n), _arrays(kind, 3 * n), _arrays(kind, 19 * n)
        capi.check(lib.hlbg_get_macro(s.ctx, _p(rho), _p(u)), s.ctx)
        capi.check(lib.hlbg_get_f(s.ctx, _p(f), 0), s.ctx)
        if kind == "odd":
            for a in (rho, u, f):
                assert a.base[0] == 7.0 and (a.base[len(a) + 1:] == 7.0).all()
        got = rho.copy(), u.copy(), f.copy(), s.WallShearStress()
        if want is None:
            want = got
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True)
