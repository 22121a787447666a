"""The frequency kernel's lane groups: 1, 2 or 3 bins per lane of half a warp (two cells at a time) up to
48 bins, 2, 4 or 8 bins per lane of a whole one beyond. Bin counts at the ends of every shape, rows
that are and are not multiples of 16 bytes, and odd numbers of cells, so that a last cell runs alone,
against the oracle."""
import numpy as np
import pytest

from helpers import matched_pair, norm_err
from lydion_b200 import workloads as W
from lydion_b200._lib import PREC_FP32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_nu", [4, 14, 16, 18, 30, 32, 34, 46, 48, 50, 64, 66, 128])
@pytest.mark.parametrize("nr,nz", [(3, 3), (7, 5), (13, 16)])
def test_steps_match_oracle(oracle_mod, n_nu, nr, nz):
    """Three full steps: J and H to 1e-9 of their maxima (the conditioning of the frequency systems),
    windows exact, the records to 1e-9."""
    cl = W.small_cloud(nr=nr, nz=nz, n_nu=n_nu, x_max=300.0, tau0=1e6)
    st, ctx = matched_pair(oracle_mod, cl, seed=5)
    h = ctx.static_steps(3, cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    d = st.run(3)
    np.testing.assert_array_equal(h[:, 5:7], d[:, 5:7])
    np.testing.assert_allclose(h[:, :5], d[:, :5], rtol=1e-9, atol=1e-9 * np.abs(d[:, 0]).max())
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < 1e-9, f
    ctx.close()


@pytest.mark.parametrize("n_nu", [12, 27, 40, 64])
def test_separate_phases_and_old_state(oracle_mod, n_nu):
    """Emission/absorption and the frequency update on their own, from a J_old that is not J (its rows are
    read beside the staged ones)."""
    n_even = n_nu + n_nu % 2
    cl = W.small_cloud(nr=9, nz=7, n_nu=n_even, x_max=300.0, tau0=1e5)
    st, ctx = matched_pair(oracle_mod, cl, seed=8)
    old = 0.7 * st.J
    st.J_old[...] = old
    ctx.upload("J_old", old)
    st.emission_absorption(cl.c_tilde, cl.dt)
    ctx.emission_absorption(cl.c_tilde, cl.dt)
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < 1e-13, f
    old = 1.1 * st.J
    st.J_old[...] = old
    ctx.upload("J_old", old)
    ctdt = cl.c_tilde * cl.dt
    st.frequency_update(ctdt)
    ctx.frequency_update(ctdt)
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < 1e-9, f
    ctx.close()


def _odd_cloud(n_nu, nr, nz, tau0=1e6):
    """A cloud of an odd number of bins: the symmetric grid of one bin more without its lowest."""
    from lydion_b200 import grid as G
    even = G.symmetric_frequency_grid(n_nu + 1, x_max=300.0)
    return W.small_cloud(nr=nr, nz=nz, n_nu=n_nu, freq=G._finish_freq_grid(even.nu[1:]), tau0=tau0)


@pytest.mark.parametrize("n_nu", [5, 15, 17, 31, 33, 47, 49, 63, 65, 127])
@pytest.mark.parametrize("nr,nz", [(7, 5), (13, 16)])
def test_odd_bins_match_oracle(oracle_mod, n_nu, nr, nz):
    """Rows of an odd number of FP64 bins, every second of which starts off a 16-byte boundary: the copies
    that go element by element. Bounds as above."""
    cl = _odd_cloud(n_nu, nr, nz)
    st, ctx = matched_pair(oracle_mod, cl, seed=6)
    h = ctx.static_steps(3, cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    d = st.run(3)
    np.testing.assert_array_equal(h[:, 5:7], d[:, 5:7])
    np.testing.assert_allclose(h[:, :5], d[:, :5], rtol=1e-9, atol=1e-9 * np.abs(d[:, 0]).max())
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < 1e-9, f
    ctx.close()


@pytest.mark.parametrize("n_nu", [6, 14, 18, 30, 34, 46, 50, 5, 17, 33, 47, 65])
def test_fp32_storage_rows_off_16_bytes(oracle_mod, n_nu):
    """FP32 rows that are no multiple of 16 bytes, against the FP64 oracle: three steps within the FP32
    form's 1e-4 of each field's maximum, where a bin read from another's place is off by tens of percent."""
    cl = _odd_cloud(n_nu, 13, 7, tau0=1e5) if n_nu % 2 else W.small_cloud(nr=13, nz=7, n_nu=n_nu, x_max=300.0, tau0=1e5)
    st, ctx = matched_pair(oracle_mod, cl, seed=6, precision=PREC_FP32)
    ctx.static_steps(3, cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    st.run(3)
    for f in ("J", "H_r", "H_Z"):
        assert norm_err(ctx.download(f), getattr(st, f)) < 1e-4, f
    ctx.close()
