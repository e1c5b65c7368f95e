"""The FP64 update on states outside the fast collision's range (densities that are
zero, negative, subnormal or not finite, distributions that are NaN or infinite),
against the oracle: the same bits, NaN and infinities in the same places."""
import numpy as np
import pytest

from hemelb_gb300 import capi, cases
from oracle.oracle import OracleLBM

pytestmark = pytest.mark.gpu

SPECIAL = (np.nan, np.inf, -np.inf, 0.0, -0.0, 1.0e308, -1.0e308, 1.0e160, 5.0e-324, 1.0e-310, -0.7)


@pytest.mark.parametrize("kernel", [capi.KERNEL_LBGK, capi.KERNEL_TRT])
def test_fp64_update_matches_oracle_on_extreme_states(kernel):
    c = cases.bifurcation(seed=5, parent_radius=6.0, parent_length=30.0, daughter_length_factor=1.2, period=100.0)
    c.params.kernel = kernel
    o = OracleLBM(c.geometry.view, c.params, c.inlets, c.outlets)
    o.set_equilibrium()
    o.step(20)
    f = o.fold().copy()
    rng = np.random.default_rng(3)
    f *= 1.0 + 0.2 * rng.standard_normal(f.shape)
    n = len(f)
    for k, v in enumerate(SPECIAL):  # single distributions, at sites of every kind
        for i in rng.integers(0, n, 8):
            f[i, rng.integers(0, 19)] = v
        f[rng.integers(0, n, 2)] = v  # whole sites
    f[rng.integers(0, n, 4)] *= -1.0
    f[rng.integers(0, n, 4)] *= 1.0e-300
    s = c.solver()
    s.SetInitialConditions()
    s.PutF(f, 0)
    s.PutF(f, 1)
    s.SetTimeStep(21)
    o.f_old[: n * 19] = f.reshape(-1)
    o.f_new[: n * 19] = f.reshape(-1)
    for _ in range(2):
        s.DoTimeStep(1)
        with np.errstate(all="ignore"):
            o.step(1)
        assert np.array_equal(s.GetFOld(), o.fold(), equal_nan=True)
        assert np.array_equal(s.GetFNew(), o.fnew(), equal_nan=True)
