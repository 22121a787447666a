"""The launch-shape knobs' automatic settings: they can be asked for, reported and put back."""
import numpy as np
import pytest

from helpers import random_state
from lydion_b200 import workloads as W
from lydion_b200._lib import SOLVER_THOMAS, LydionError

pytestmark = pytest.mark.gpu


def _context(cl):
    from lydion_b200.m1 import context_for_cloud
    ctx = context_for_cloud(cl)
    for name, a in zip(("J", "H_r", "H_Z"), random_state(cl, 4)):
        ctx.upload(name, a)
    return ctx


def test_automatic_knobs_stay_automatic():
    ctx = _context(W.small_cloud(nr=12, nz=10, n_nu=16))
    new = ctx.tuning()
    assert new[0] < 0 and new[1] < 0
    ctx.set_tuning(*new)                     # what was read, written back
    assert ctx.tuning() == new
    ctx.set_tuning(solver=SOLVER_THOMAS)     # one knob set, the others left to the library
    assert ctx.tuning()[:3] == (new[0], new[1], SOLVER_THOMAS)
    ctx.set_tuning(8, 16)
    assert ctx.tuning()[:2] == (8, 16)
    ctx.set_tuning(0, 0)
    assert ctx.tuning() == new
    ctx.close()


@pytest.mark.parametrize("rows,cells", [(2, 0), (-4, 0), (65, 0), (0, 7), (0, -7), (0, 1025), (0, -1025)])
def test_other_values_are_refused(rows, cells):
    ctx = _context(W.small_cloud(nr=12, nz=10, n_nu=16))
    before = ctx.tuning()
    with pytest.raises(LydionError):
        ctx.set_tuning(rows, cells)
    assert ctx.tuning() == before
    ctx.close()


def test_host_step_follows_the_tuning():
    """The automatic height depends on the CTAs per SM: the host-state step's row chunks are cut again when
    that changes between two calls."""
    cl = W.static_cloud(nr=96, nz=192, n_nu=64, tau0=1e6, T0=1e4, umax_kms=100.0, rs=0.5, tau_abs=0.5)
    dev, host = _context(cl), _context(cl)
    p = (cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)
    state = [host.download(f) for f in ("J", "H_r", "H_Z")]
    for ctas in (2, 3, 2):
        host.set_tuning(0, 0, 0, ctas)
        dev.static_steps(1, *p)
        state = list(host.static_step_host(*state, *p, chunks=3)[:3])
        for f, a in zip(("J", "H_r", "H_Z"), state):
            np.testing.assert_array_equal(a, dev.download(f), err_msg=f"{f} at {ctas} CTAs per SM")
    dev.close()
    host.close()
