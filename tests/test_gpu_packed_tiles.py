"""The packed advection tiles: the active window cut into chunks of bins and the threads dealt out
over (column, bin) pairs. Windows of one bin to all of them, at the edges of a chunk (31, 32, 33
bins), on fields narrower and wider than a tile, against the oracle's advection of the same
bins; bins outside the window pass through unchanged."""
import numpy as np
import pytest

from helpers import matched_pair, norm_err
from lydion_b200 import workloads as W
from lydion_b200._lib import PREC_FP32, PREC_MIXED

pytestmark = pytest.mark.gpu

WINDOWS = [(0, 63), (0, 0), (63, 63), (5, 11), (20, 43), (1, 31), (16, 47), (30, 62), (6, 57)]


@pytest.mark.parametrize("nr,nz,bot,flux", [(3, 3, W.BC_REFLECT, W.FLUX_GLF), (7, 33, W.BC_OUTFLOW, W.FLUX_HLL),
                                            (17, 5, W.BC_REFLECT, W.FLUX_GLF), (41, 19, W.BC_OUTFLOW, W.FLUX_GLF)])
def test_any_window_matches_oracle(oracle_mod, nr, nz, bot, flux):
    cl = W.small_cloud(nr=nr, nz=nz, n_nu=64, x_max=300.0, bc_z_bot=bot, flux_method=flux)
    ctdt = cl.c_tilde * cl.dt
    for q, (kmin, kmax) in enumerate(WINDOWS):
        st, ctx = matched_pair(oracle_mod, cl, seed=31 + q)
        before = {f: getattr(st, f).copy() for f in ("J", "H_r", "H_Z")}
        st.advect_jh(ctdt, kmin, kmax, True)
        ctx.advect_jh(ctdt, kmin, kmax, True, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
        for f in ("J", "H_r", "H_Z"):
            got = ctx.download(f)
            assert norm_err(got, getattr(st, f)) < 1e-12, (f, kmin, kmax)
            out = np.ones(cl.n_nu, dtype=bool)
            out[kmin:kmax + 1] = False
            np.testing.assert_array_equal(got[:, :, out], before[f][:, :, out])
        ctx.close()


@pytest.mark.parametrize("precision,tol", [(PREC_MIXED, 2e-6), (PREC_FP32, 2e-6)])
def test_reduced_forms_match_oracle(oracle_mod, precision, tol):
    """FP32 arithmetic: one advection is within a few FP32 roundings (2^-24 times the ~10 terms
    of a flux sum) of the field's maximum."""
    cl = W.small_cloud(nr=29, nz=23, n_nu=50, x_max=300.0, bc_z_bot=W.BC_OUTFLOW)
    ctdt = cl.c_tilde * cl.dt
    for kmin, kmax in [(0, 49), (9, 40), (24, 24)]:
        st, ctx = matched_pair(oracle_mod, cl, seed=3, precision=precision)
        st.advect_jh(ctdt, kmin, kmax, True)
        ctx.advect_jh(ctdt, kmin, kmax, True, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
        for f in ("J", "H_r", "H_Z"):
            assert norm_err(ctx.download(f), getattr(st, f)) < tol, (f, kmin, kmax)
        ctx.close()


@pytest.mark.parametrize("rows", [4, 5, 16, 64])
def test_tile_heights_change_nothing(oracle_mod, rows):
    """Tiles of a set height and the heights the library picks give the same bits."""
    cl = W.small_cloud(nr=37, nz=27, n_nu=48, x_max=200.0)
    _, a = matched_pair(oracle_mod, cl, seed=11)
    _, b = matched_pair(oracle_mod, cl, seed=11)
    b.set_tuning(rows)
    for ctx in (a, b):
        ctx.static_steps(5, cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    for f in ("J", "H_r", "H_Z"):
        np.testing.assert_array_equal(a.download(f), b.download(f))
    a.close()
    b.close()


@pytest.mark.parametrize("staging", [0, 2])
def test_repeated_band_advections_keep_the_old_state(oracle_mod, staging):
    """AdvectJandH! again and again from a J_old that is not J: the buffers trade places, J_old stays, and
    a fused step afterwards (with tensor maps or without) starts from the advected state."""
    cl = W.small_cloud(nr=17, nz=11, n_nu=24, x_max=200.0)
    st, ctx = matched_pair(oracle_mod, cl, seed=13)
    ctx.set_tuning(8, 0, 0, 0, staging)
    ctdt = cl.c_tilde * cl.dt
    old = 0.5 * st.J
    st.J_old[...] = old
    ctx.upload("J_old", old)
    for n in range(4):
        st.advect_jh(ctdt, 0, 23, n == 3)
        ctx.advect_jh(ctdt, 0, 23, n == 3, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
        for f in ("J", "H_r", "H_Z", "J_old"):
            assert norm_err(ctx.download(f), getattr(st, f)) < 4e-12, (n, f)
    h = ctx.static_steps(2, cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    d = st.run(2)
    np.testing.assert_array_equal(h[:, 5:7], d[:, 5:7])
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < 1e-9, f
    ctx.close()
