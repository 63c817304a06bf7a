"""Grid sums of the CG and BiCGStab kernels at the block counts where their path changes: a
box of two blocks, the last count whose final block adds the partials itself
(1216), the first that leaves them to a kernel of its own, and a count on
a grid of wide rows.  The right-hand side's norm (one sum and, for the
closed box, a mean) to 1e-13: at most some hundred roundings of 1.1e-16 lie
between a term and its sum.  The solve's own residual norm by the reference's
matrix."""
import numpy as np
import pytest

from simcoflow3d_gb300 import capi, geometry as GM, predictor as PR, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# 2, 1216, 1232 and 1320 blocks of 32 x 4 columns, 2 (the last: 8) cells along k
SHAPES = [(8, 4, 4), (32, 64, 152), (32, 64, 153), (160, 130, 64)]


@pytest.mark.parametrize("closed", [True, False])
@pytest.mark.parametrize("precision,tol", [(0, 1e-10), (1, 1e-8)])
@pytest.mark.parametrize("shape", SHAPES)
def test_grid_sums(gpu_lib, shape, precision, tol, closed):
    from simcoflow3d_gb300.projection import Projection
    w = W.build_workload("sums", *shape, liquid=("bubble", 0.5, 0.5, 0.6, 0.2), rho_l=1000.0, rho_g=1.2,
                         extent=tuple((0.0, n / 32.0) for n in shape), bcp_flag=(1, 1, 1, 1, 1, int(closed)))
    pc = O.pocoef(w)
    A, b = O.csr(w, pc), O.rhs(w, pc)
    pos = w.arrays["posnu"]
    act = pos >= 0
    p = Projection.for_workload(w, rel_tol=tol, precision=precision)
    _, pp, st = p.poisson_solve(w)
    bc = b - b.mean() if closed else b
    assert abs(st["rhs_norm"] - np.linalg.norm(bc)) <= 1e-13 * np.linalg.norm(bc)
    x = np.zeros(w.ext_cell + 1)
    x[pos[act]] = pp[1:-1, 1:-1, 1:-1][act]
    # the recomputed FP64 residual rounds once more than the solver's own
    assert st["converged"] == 1 and O.csr_relres(A, b, x, closed) <= tol * (1 + 1e-3)
    p.close()


# 8, 1377 and 2745 blocks: every pass's last block sums, P's and S's alone, none
@pytest.mark.parametrize("I,J,K", [(9, 7, 4), (3, 609, 129), (3, 1217, 129)])
@pytest.mark.parametrize("precision", [capi.SCF_PREC_FP64, capi.SCF_PREC_MIXED])
def test_predictor_sums(gpu_lib, I, J, K, precision):
    """Dp bit for bit; the velocities of two solves to a residual of 1e-12 agree
    to 1e-12 times the Jacobi-scaled systems' condition, a few hundred by the
    109 iterations of the longest box: 1e-9 (relative L2)."""
    g = O.grid_preprocess(GM.geometry_inputs("box", shape=(I, J, K), solid=W.SPHERE_C1))
    inp = PR.momentum_inputs(g, vof_old_noise=0.01)
    opts = PR.default_opts(precision=precision, rel_tol=1e-12)
    po, do, _ = O.predict_solves(inp, opts)
    pg, dg, _ = PR.PredictSolves(I, J, K)(inp, opts)
    for c in range(3):
        assert np.array_equal(dg[c], do[c])
        assert np.linalg.norm(pg[c] - po[c]) <= 1e-9 * np.linalg.norm(po[c])
