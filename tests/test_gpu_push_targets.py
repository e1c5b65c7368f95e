"""Where the update's pushes land when blocks around a block are missing: random fluid
masks over blocks that are there or not, so that boundary sites meet a block across an
edge without the one across the face, and blocks of one z column with gaps."""
import ctypes as C

import numpy as np
import pytest

from hemelb_gb300 import capi
from hemelb_gb300.lbm import LBM, LbmParameters
from oracle.oracle import OracleLBM

pytestmark = pytest.mark.gpu

CX = [1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
CY = [0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1]
CZ = [0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1]


def sparse_geometry(seed, shape, fill):
    """Wall links at every fluid site beside a solid or missing one."""
    rng = np.random.default_rng(seed)
    there = rng.random(shape) < 0.6
    there[0, 0, 0] = there[-1, -1, -1] = True
    coords = np.argwhere(there).astype(np.int32)
    coords = coords[rng.permutation(len(coords))]
    fluid = rng.random((len(coords), 8, 8, 8)) < fill
    fluid[0] = True
    dense = np.zeros([8 * n + 2 for n in shape], dtype=bool)
    for (x, y, z), m in zip(coords, fluid):
        dense[8 * x + 1: 8 * x + 9, 8 * y + 1: 8 * y + 9, 8 * z + 1: 8 * z + 9] = m
    sites = np.argwhere(fluid.reshape(-1))[:, 0]
    at = coords[sites >> 9] * 8 + np.stack([(sites >> 6) & 7, (sites >> 3) & 7, sites & 7], axis=1) + 1
    wall = np.zeros(len(sites), dtype=np.uint32)
    for d in range(18):
        wall |= np.where(dense[at[:, 0] + CX[d], at[:, 1] + CY[d], at[:, 2] + CZ[d]], 0, 1 << d).astype(np.uint32)
    edge = wall != 0
    n = int(edge.sum())
    keep = dict(block_coords=np.ascontiguousarray(coords),
                fluid_mask=np.packbits(fluid.reshape(-1, 64), axis=1, bitorder="little").view(np.uint64).copy(),
                link_site=sites[edge].astype(np.int64), wall_mask=wall[edge].copy(),
                iolet_mask=np.zeros(n, np.uint32), iolet_id=np.full(n, -1, np.int32),
                site_type=np.ones(n, np.int8), cut_distance=rng.uniform(0.01, 0.99, (n, 18)).astype(np.float32))
    g = capi.Geometry()
    g.q, g.block_size, g.n_blocks, g.n_link_sites = 19, 8, len(coords), n
    g.blocks[:] = shape
    types = dict(capi.Geometry._fields_)
    for k, v in keep.items():
        setattr(g, k, C.cast(v.ctypes.data, types[k]))
    g._keep = keep
    return g


def start(n, seed):
    rng = np.random.default_rng(seed)
    return 1.0 + 0.02 * rng.standard_normal(n), 0.02 * rng.standard_normal((n, 3))


@pytest.mark.parametrize("fill", [0.55, 0.97])
@pytest.mark.parametrize("variant", [1, 6])
def test_pushes_across_missing_blocks_fp64_bit_exact(fill, variant):
    g = sparse_geometry(11, (3, 3, 4), fill)
    p = LbmParameters(tau=0.8, precision=capi.FP64)
    s = LBM(g, p)
    rho, u = start(s.n_sites, 5)
    s.SetInitialField(rho, u)
    s.SetLaunchVariant(variant)
    o = OracleLBM(g, p, [], [])
    f = s.GetFOld()
    o.set_equilibrium()
    o.f_old[: f.size] = f.reshape(-1)
    o.f_new[: f.size] = s.GetFNew().reshape(-1)
    s.DoTimeStep(3)
    o.step(3)
    assert np.array_equal(s.GetFOld(), o.fold())


@pytest.mark.parametrize("fill", [0.3, 0.55, 0.97])
@pytest.mark.parametrize("variant", [1, 6])
def test_gathered_interpolated_links_fp64_bit_exact(fill, variant):
    """BFL walls: from no interpolated link in a warp to several hundred."""
    g = sparse_geometry(13, (2, 3, 3), fill)
    p = LbmParameters(tau=0.8, precision=capi.FP64, wall=capi.WALL_BFL)
    for monitored in (False, True):
        s = LBM(g, p)
        rho, u = start(s.n_sites, 7)
        s.SetInitialField(rho, u)
        s.SetLaunchVariant(variant)
        f = s.GetFOld()
        o = OracleLBM(g, p, [], [])
        o.set_equilibrium()
        o.f_old[: f.size] = f.reshape(-1)
        o.f_new[: f.size] = s.GetFNew().reshape(-1)
        if monitored:
            for _ in range(3):
                s.StepMonitored(1)
        else:
            s.DoTimeStep(3)
        o.step(3)
        assert np.array_equal(s.GetFOld(), o.fold())


@pytest.mark.parametrize("precision", [capi.FP32DEV, capi.FP16])
@pytest.mark.parametrize("fill", [0.55, 0.97])
def test_pushes_and_monitored_lookups_give_the_same_distributions(precision, fill):
    g = sparse_geometry(12, (4, 2, 3), fill)
    got = []
    for variant, monitored in ((6, True), (6, False), (5, False), (0, False), (4, False), (8, False)):
        s = LBM(g, LbmParameters(tau=0.8, precision=precision))
        rho, u = start(s.n_sites, 6)
        s.SetInitialField(rho, u)
        s.SetLaunchVariant(variant)
        if monitored:
            for _ in range(3):
                s.StepMonitored(1)
        else:
            s.DoTimeStep(3)
        got.append(s.GetFOld())
        s.close()
    for other in got[1:]:
        assert np.array_equal(got[0], other)
