"""Where the fused StabilityTester's partials are folded: inside the update's launch, or,
from 256 CTAs on, by a launch of their own behind it.  Boxes of full blocks give CTA
counts on both sides of the line and remainders of the fold's own CTAs; the stats of each
step are compared with the separate reduction of a twin that makes plain steps."""
import ctypes as C
import time

import numpy as np
import pytest

from hemelb_gb300 import capi, cases
from hemelb_gb300.lbm import LBM, LbmParameters
from tests.test_gpu_push_targets import CX, CY, CZ, start

pytestmark = pytest.mark.gpu



def box(blocks, side=4):
    """`blocks` blocks of a box `side` blocks wide in y and z, all fluid, walls around."""
    b = np.arange(blocks)
    coords = np.stack([b // (side * side), b // side % side, b % side], axis=1).astype(np.int32)
    shape = coords.max(axis=0) + 1
    there = np.zeros(shape + 2, dtype=bool)
    there[coords[:, 0] + 1, coords[:, 1] + 1, coords[:, 2] + 1] = True
    l = np.arange(512)
    local = np.stack([l >> 6, (l >> 3) & 7, l & 7], axis=1)
    wall = np.zeros((blocks, 512), dtype=np.uint32)
    for d in range(18):
        step = local + np.array([CX[d], CY[d], CZ[d]])
        cell = (step >> 3) + 1  # 0, 1 or 2: the block it is in
        for c in np.unique(cell, axis=0):
            at = coords + c
            missing = ~there[at[:, 0], at[:, 1], at[:, 2]]
            wall[np.ix_(missing, (cell == c).all(axis=1))] |= np.uint32(1 << d)
    wall = wall.reshape(-1)
    edge = np.flatnonzero(wall)
    keep = dict(block_coords=coords, fluid_mask=np.full((blocks, 8), ~np.uint64(0), dtype=np.uint64),
                link_site=edge.astype(np.int64), wall_mask=wall[edge].copy(),
                iolet_mask=np.zeros(len(edge), np.uint32), iolet_id=np.full(len(edge), -1, np.int32),
                site_type=np.ones(len(edge), np.int8))
    g = capi.Geometry()
    g.q, g.block_size, g.n_blocks, g.n_link_sites = 19, 8, blocks, len(edge)
    g.blocks[:] = [int(n) for n in shape]
    types = dict(capi.Geometry._fields_)
    for k, v in keep.items():
        setattr(g, k, C.cast(v.ctypes.data, types[k]))
    g._keep = keep
    return g


# CTAs of a full block: FP64 16 of one warp in the list (6) and 4 of 128 slots (1); FP32
# and FP16 4 in either
@pytest.mark.parametrize("precision,variant,blocks", [
    (capi.FP64, 6, 15), (capi.FP64, 6, 16), (capi.FP64, 6, 17), (capi.FP64, 6, 31), (capi.FP64, 6, 32), (capi.FP64, 6, 33), (capi.FP64, 6, 70),
    (capi.FP64, 1, 63), (capi.FP64, 1, 64), (capi.FP64, 1, 127), (capi.FP64, 1, 128),
    (capi.FP32DEV, 6, 1), (capi.FP32DEV, 6, 63), (capi.FP32DEV, 1, 64), (capi.FP32DEV, 6, 65), (capi.FP32DEV, 6, 127), (capi.FP32DEV, 6, 128), (capi.FP32DEV, 6, 129),
    (capi.FP32DEV, 3, 300), (capi.FP16, 2, 257), (capi.FP16, 5, 400)])
def test_stats_of_every_step_on_both_sides_of_the_line(precision, variant, blocks):
    g = box(blocks)
    a, b = LBM(g, LbmParameters(tau=0.8, precision=precision)), LBM(g, LbmParameters(tau=0.8, precision=precision))
    rho, u = start(a.n_sites, blocks)
    for s in (a, b):
        s.SetInitialField(rho, u)
        s.SetLaunchVariant(variant)
    assert a.StepMonitored(1).time_step == -1
    for k in range(1, 5):
        sa = a.StepMonitored(1)
        b.DoTimeStep(1)
        sb = b.reduce()
        rho, u = b.macro()
        inc = a.Incompressibility()
        assert sa.time_step == sb.time_step == k + 1
        assert sa.unstable_sites == sb.unstable_sites
        if precision == capi.FP64:
            assert sa.max_du == sb.max_du and sa.min_f == sb.min_f
            assert abs(sa.mass - sb.mass) <= 1e-12 * sb.mass
            assert abs(inc.min_density - rho.min()) <= 1e-14 and abs(inc.max_density - rho.max()) <= 1e-14
        else:
            assert abs(sa.max_du - sb.max_du) <= 1e-5 * sb.max_du + 1e-12
            assert abs(sa.min_f - sb.min_f) <= 1e-6 and abs(sa.mass - sb.mass) <= 1e-9 * sb.mass
            assert abs(inc.min_density - rho.min()) <= 1e-6 and abs(inc.max_density - rho.max()) <= 1e-6
    # the same run again, and in one call: the same numbers to the last bit
    for calls in (5, 1):
        b.SetInitialField(*start(a.n_sites, blocks))
        b.SetTimeStep(1)
        for _ in range(calls):
            sb = b.StepMonitored(5 // calls)
        assert (sa.mass, sa.max_du, sa.min_f) == (sb.mass, sb.max_du, sb.min_f)


@pytest.mark.parametrize("blocks", [8, 40])
def test_nan_reaches_the_stats(blocks):
    g = box(blocks)
    a, b = LBM(g, LbmParameters(tau=0.8, precision=capi.FP64)), LBM(g, LbmParameters(tau=0.8, precision=capi.FP64))
    a.SetInitialConditions()
    f = a.GetFOld()
    f[11] = np.nan
    for s in (a, b):
        s.SetInitialConditions()
        s.PutF(f, 0)
    a.StepMonitored(1)
    sa = a.StepMonitored(1)
    b.DoTimeStep(1)
    sb = b.reduce()
    assert sa.unstable_sites == sb.unstable_sites > 0 and sa.min_f == sb.min_f
    assert np.isnan(sa.max_du) and np.isnan(sa.mass)


def test_a_checked_step_of_a_large_run_costs_little_more_than_a_plain_one():
    """The velocities a check reads and writes are 24 bytes a site beside the update's
    152, and the step's time went from 7.55 to 9.51 ms with them on a vascular forest
    (26 %) when the partials had launches of their own.  Here it is 29 %, and was 45 % when
    the update's CTAs folded them; half way is the line."""
    s = cases.tree(7, 512, 1, 6, 50.0, precision=capi.FP32DEV).solver()
    s.SetInitialConditions()
    s.SetLaunchVariant(6)
    s.DoTimeStep(5)
    plain = min(s.time_steps(40) for _ in range(5)) / 40
    s.StepMonitored(5)
    checked = []
    for _ in range(5):
        t = time.perf_counter()
        s.StepMonitored(40)
        checked.append((time.perf_counter() - t) / 40 * 1e3)
    assert min(checked) < 1.37 * plain
