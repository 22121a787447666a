"""The adjoint on fields of more cells than one wave of its frequency kernel has warps (2368 on 148
SMs), where a warp takes several cells and the last CTA is part full, against the dual-number
build of the oracle. A cell left out or taken twice changes a directional derivative by about one part
in the number of cells (4e-4 here); the rounding of the two stiff solves stays within 1e-8 on the
10 x 9 field, so 1e-6 separates the two with two decades on either side."""
import numpy as np
import pytest

import test_gpu_adjoint as A
from lydion_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz,nnu", [(61, 53, 16), (41, 59, 40)])
def test_many_cells_match_forward_mode_oracle(oracle_mod, monkeypatch, nr, nz, nnu):
    monkeypatch.setattr(A, "_cloud", lambda flux: W.small_cloud(nr=nr, nz=nz, n_nu=nnu, flux_method=flux))
    P = A.Problem(2)
    ctx, g = P.adjoint(every=1)
    ctx.close()
    cl = P.cl
    st = oracle_mod.OracleState(cl)
    for name, a in zip(("J", "H_r", "H_Z"), P.state):
        getattr(st, name)[...] = a
        getattr(st, name + "_old")[...] = a
    st.setup_profiles()
    rng = np.random.default_rng(23)
    for key, v in (("alpha", cl.alpha), ("T", cl.T), ("J0", P.state[0])):
        sd = rng.uniform(0.5, 1.5, size=v.shape) * v
        obj, tan, _, _ = oracle_mod.objective_tangent(st, P.n, 1.0, A.SS * P.w, {key: sd})
        assert obj == pytest.approx(g["objective"], rel=1e-10)
        assert float(np.sum(g["grad_" + key] * sd)) == pytest.approx(tan, rel=1e-6), key
