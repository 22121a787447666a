"""static_steps replays a captured graph of four steps once a context has run 64, and launches the steps
left over one by one. Calls of at most three steps never replay: a context that only makes such calls
is the reference, bit for bit, for one that crosses the threshold, leaves remainders, or has an input
appear, change or go between two replayed stretches."""
import numpy as np
import pytest

from helpers import random_state
from lydion_b200 import workloads as W
from lydion_b200._lib import PREC_FP32, PREC_FP64

pytestmark = pytest.mark.gpu


def _cloud():
    return W.small_cloud(nr=9, nz=7, n_nu=32, x_max=300.0, tau0=1e5)


def _context(cl, precision=PREC_FP64):
    from lydion_b200.m1 import context_for_cloud
    ctx = context_for_cloud(cl, precision=precision)
    for name, a in zip(("J", "H_r", "H_Z"), random_state(cl, 4)):
        ctx.upload(name, a)
    return ctx


def _steps(ctx, cl, calls):
    return np.concatenate([ctx.static_steps(n, cl.c_tilde, cl.dt, cl.z_center, cl.bc_r_right, cl.bc_z_bot,
                                            cl.bc_z_top) for n in calls])


def _direct(ctx, cl, n):
    return _steps(ctx, cl, [3] * (n // 3) + ([n % 3] if n % 3 else []))


def _same(a, b):
    for f in ("J", "H_r", "H_Z"):
        np.testing.assert_array_equal(a.download(f), b.download(f), err_msg=f)
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32])
def test_thresholds_and_remainders(precision):
    cl = _cloud()
    a, b = _context(cl, precision), _context(cl, precision)
    np.testing.assert_array_equal(_steps(a, cl, (63, 1, 7, 66)), _direct(b, cl, 137))
    _same(a, b)


def _alpha_cF(ctx, cl):
    ctx.upload("alpha_cF", 0.3 * cl.alpha * np.linspace(0.5, 1.5, cl.nr)[None, :])


def _alpha_F(ctx, cl):
    rng = np.random.default_rng(6)
    ctx.upload("alpha_F", cl.alpha.mean() * 1e-3 * rng.uniform(0.5, 2.0, size=(cl.nz, cl.nr, cl.n_nu)))


def _phi_nu(ctx, cl):
    rng = np.random.default_rng(7)
    phi = rng.uniform(0.5, 1.5, size=(cl.nz, cl.nr, cl.n_nu))
    ctx.upload("phi_nu", phi / (phi * cl.freq.dnu).sum(axis=2, keepdims=True))


def _phi_range(ctx, cl):
    ctx.update_phi_nu(0, cl.n_nu - 1)


def _advect_jh(ctx, cl):
    ctx.upload("J_old", ctx.download("J"))
    ctx.advect_jh(cl.c_tilde * cl.dt, 0, cl.n_nu - 1, False, cl.bc_r_right, cl.bc_z_bot, cl.bc_z_top)


def _tuning(ctx, cl):
    ctx.set_tuning(4, 8, 1)


@pytest.mark.parametrize("before,change", [((), (_alpha_cF,)), ((), (_alpha_F,)), ((), (_phi_nu,)), ((), (_phi_range,)),
                                           ((_phi_nu,), (_phi_range,)), ((), (_advect_jh,)), ((), (_tuning,)),
                                           ((_phi_nu,), (_alpha_F, _phi_range, _alpha_cF, _advect_jh))],
                         ids=lambda fs: "+".join(f.__name__[1:] for f in fs) or "none")
def test_inputs_changed_between_replays(before, change):
    cl = _cloud()
    a, b = _context(cl), _context(cl)
    for ctx in (a, b):
        for f in before:
            f(ctx, cl)
    np.testing.assert_array_equal(_steps(a, cl, (68,)), _direct(b, cl, 68))
    for ctx in (a, b):
        for f in change:
            f(ctx, cl)
    np.testing.assert_array_equal(_steps(a, cl, (7, 4)), _direct(b, cl, 11))
    _same(a, b)
