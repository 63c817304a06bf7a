"""The momentum rows' shortcuts (csrc/k_predictor.cu) against the oracle: rows
with and without convective terms, densities that are powers of two and not,
gravity along and across the component, a time step whose quotients leave the
range of the reciprocal division.  Dp bit for bit; the solve to a residual of
1e-12, so its velocities to 1e-9 (relative L2) on these well-conditioned
boxes."""
import numpy as np
import pytest

from simcoflow3d_gb300 import capi, geometry as GM, predictor as PR, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

OPTIONS = [dict(), dict(rho_w_ref=1000.0, rho_a_ref=1.2), dict(rho_w_ref=1.0, rho_a_ref=0.25, dt=0.125),
           dict(gx=0.3, gy=-9.81, gz=0.0), dict(gz=-0.0, g=-9.81), dict(beta_vis=1.0), dict(dt=1.3 * 2.0 ** -310)]


@pytest.mark.parametrize("noise", [0.0, 0.01])
@pytest.mark.parametrize("kw", OPTIONS)
def test_rows_match_oracle(gpu_lib, kw, noise):
    shape = (14, 11, 12)
    g = O.grid_preprocess(GM.geometry_inputs("box", shape=shape, solid=W.SPHERE_C1))
    inp = PR.momentum_inputs(g, vof_old_noise=noise)
    opts = PR.default_opts(precision=capi.SCF_PREC_FP64, rel_tol=1e-12)
    for name, value in kw.items():
        setattr(opts, name, value)
    po, do, _ = O.predict_solves(inp, opts)
    pg, dg, _ = PR.PredictSolves(*shape)(inp, opts)
    for c in range(3):
        assert np.array_equal(dg[c], do[c])
        assert np.linalg.norm(pg[c] - po[c]) <= 1e-9 * np.linalg.norm(po[c])
