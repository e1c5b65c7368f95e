"""Every launch shape of the FP32 and FP16 updates, plain and monitored, against the
slot-list kernel of the per-range calls, which looks its neighbours up site by site and
dispatches its links one by one: random masks over blocks with gaps, both kinds of wall."""
import numpy as np
import pytest

from hemelb_gb300 import capi
from hemelb_gb300.lbm import LBM, LbmParameters
from tests.test_gpu_push_targets import sparse_geometry, start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.FP32DEV, capi.FP16])
@pytest.mark.parametrize("fill", [0.3, 0.55, 0.97])
@pytest.mark.parametrize("wall", [capi.WALL_SBB, capi.WALL_BFL])
def test_every_shape_against_the_slot_list(precision, fill, wall):
    g = sparse_geometry(23, (4, 2, 3), fill)

    def solver():
        s = LBM(g, LbmParameters(tau=0.8, precision=precision, wall=wall))
        s.SetInitialField(*start(s.n_sites, 8))
        return s

    ref = solver()
    for _ in range(3):
        ref.StreamAndCollide(0, ref.n_sites)
        ref.PostStep(0, ref.n_sites)
        ref.SwapOldAndNew()
    want = ref.GetFOld()
    # three steps: an FP32 collision rounds a value of at most 1/3 some ten times by 2^-25
    # of it, an FP16 store a deviation of at most 0.1 by 2^-11 of it; a wrong target or
    # link is off by 0.01
    tol = 3 * 10 * 2.0 ** -25 if precision == capi.FP32DEV else 3 * 0.1 * 2.0 ** -11
    assert 20 * tol < 0.01
    for variant, monitored in [(v, False) for v in range(9)] + [(1, True), (2, True), (3, True), (6, True)]:
        s = solver()
        s.SetLaunchVariant(variant)
        if monitored:
            for _ in range(3):
                s.StepMonitored(1)
        else:
            s.DoTimeStep(3)
        assert np.abs(s.GetFOld() - want).max() <= tol, (variant, monitored)
        s.close()
