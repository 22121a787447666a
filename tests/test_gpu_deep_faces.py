"""Faces of extreme optical depth: the flux of a face is the diffusive one alone, and H feels the mean
pressure of the two sides, whatever the depth. FP32 arithmetic has to hold that far beyond the depth whose
square leaves its range (tau = 1.8e19), as the FP64 oracle does."""
import numpy as np
import pytest

from helpers import matched_pair, norm_err
from lydion_b200 import workloads as W
from lydion_b200._lib import PREC_FP32, PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(PREC_FP64, 1e-12), (PREC_MIXED, 2e-6), (PREC_FP32, 2e-6)])
@pytest.mark.parametrize("flux", [W.FLUX_GLF, W.FLUX_HLL])
@pytest.mark.parametrize("depth", [1e8, 0.9e18, 1.1e18, 1e19, 1e25, 8e37, 3e38])
def test_advection_at_depth_matches_oracle(oracle_mod, depth, flux, precision, tol):
    """One advection of an explicit alpha_F that gives the deepest faces tau = `depth`. A few FP32
    roundings (2^-24 times the ~10 terms of a flux sum) of the field's maximum, and 1e-12 in FP64."""
    cl = W.small_cloud(nr=19, nz=13, n_nu=24, x_max=200.0, bc_z_bot=W.BC_OUTFLOW, flux_method=flux)
    st, ctx = matched_pair(oracle_mod, cl, seed=17, precision=precision)
    g = cl.geom
    widest = max(np.max(a) for a in (g.dr_L + g.dr_R, g.dZ_L + g.dZ_R, g.dr_b[[0, 5]] + g.dr_b[[1, 6]],
                                     g.dZ_b[[0, 5]] + g.dZ_b[[1, 6]]))
    alpha_F = np.full((cl.nz, cl.nr, cl.n_nu), depth / widest)
    st.alpha_F[...] = alpha_F
    ctx.upload("alpha_F", alpha_F)
    ctdt = cl.c_tilde * cl.dt
    st.advect_jh(ctdt, 0, cl.n_nu - 1, True)
    ctx.advect_jh(ctdt, 0, cl.n_nu - 1, True, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < tol, f
    ctx.close()
