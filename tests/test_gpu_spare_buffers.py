"""AdvectJandH! with J_old apart from J writes a third set of J, H_r, H_Z buffers, which the context keeps between
such calls and gives back when an adjoint run wants the memory."""
import gc

import pytest

from helpers import matched_pair, norm_err
from lydion_b200 import workloads as W
from lydion_b200._lib import LydionError

pytestmark = pytest.mark.gpu


def test_an_adjoint_run_gets_the_spare_set_s_memory(oracle_mod):
    import torch
    cl = W.small_cloud(nr=128, nz=96, n_nu=64, x_max=300.0)
    st, ctx = matched_pair(oracle_mod, cl, seed=3)
    ctdt, field = cl.c_tilde * cl.dt, 8 * cl.nr * cl.nz * cl.n_nu

    def advect():
        st.advect_jh(ctdt, 0, cl.n_nu - 1, False)
        ctx.advect_jh(ctdt, 0, cl.n_nu - 1, False, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
        for f in ("J", "H_r", "H_Z", "J_old"):
            assert norm_err(ctx.download(f), getattr(st, f)) < 4e-12, f

    free = lambda: torch.cuda.mem_get_info(0)[0]
    gc.collect()                                  # (no other test's context goes while this one counts)
    for f in ("J", "H_r", "H_Z", "J_old"):
        ctx.download(f)                           # (the staging buffers are there before the count)
    none = free()
    advect()
    held = free()
    assert none - held >= 3 * field
    # a workspace of 20000 kept steps, 7 fields each: more than any GPU has
    with pytest.raises(LydionError):
        ctx.adjoint(20000, cl.c_tilde, cl.dt, cl.z_center, checkpoint_every=1)
    # the record history of those steps stays (1.1 MB, in the allocator's granules of 2 MB)
    assert free() - held >= 3 * field - (4 << 20)
    advect()                                      # allocated again
    ctx.close()
