"""Column segments of every length the launch rules choose (2 to 32 cells per
thread along k), on boxes whose extents leave remainders in every direction:
the projection's assembly bit for bit and its solve by the reference's matrix,
the predictor and the geometry against the oracle."""
import numpy as np
import pytest

from simcoflow3d_gb300 import capi, geometry as GM, predictor as PR, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# solver / assembly segment lengths: 2/4, 4/8, 8/16, 16/32
BOXES = [(70, 45, 35), (100, 90, 61), (130, 120, 75), (200, 150, 70)]


@pytest.mark.parametrize("I,J,K", BOXES)
def test_projection_segments(gpu_lib, I, J, K):
    from simcoflow3d_gb300.projection import Projection
    w = W.build_workload("box", I, J, K, solid=W.SPHERE_C1, liquid=W._surface(0.5, 0.02, None), perturb_vof_old=0.01)
    pc = O.pocoef(w)
    A, b = O.csr(w, pc), O.rhs(w, pc)
    pos = w.arrays["posnu"]
    act = pos >= 0
    rows = np.repeat(np.arange(w.ext_cell + 1), np.diff(A[0]))
    own = A[1][:rows.size] == rows
    for precision, tol in ((0, 1e-10), (1, 1e-8)):
        p = Projection.for_workload(w, rel_tol=tol, precision=precision)
        got, pp, st = p.poisson_solve(w)
        assert np.array_equal(got, pc, equal_nan=True)
        op = p.debug_operator()
        assert np.array_equal(op["diag"][act], A[2][:rows.size][own][pos[act]])
        assert st["converged"] == 1
        x = np.zeros(w.ext_cell + 1)
        x[pos[act]] = pp[1:-1, 1:-1, 1:-1][act]
        # the recomputed FP64 residual rounds once more than the solver's own
        assert O.csr_relres(A, b, x, True) <= tol * (1 + 1e-3)
        p.close()
    p = Projection.for_workload(w)
    p.stage(w, correction=False)
    assert np.array_equal(p.debug_operator()["rhs"][act], b[pos[act]])   # before the solve removes the mean


@pytest.mark.parametrize("I,J,K", [(67, 53, 75), (130, 126, 60)])
def test_predictor_segments(gpu_lib, I, J, K):
    """Solver segments of 4 and 8 cells, assembly segments of 2 and 4."""
    g = O.grid_preprocess(GM.geometry_inputs("box", shape=(I, J, K), solid=W.SPHERE_C1))
    inp = PR.momentum_inputs(g, vof_old_noise=0.01)
    opts = PR.default_opts(precision=capi.SCF_PREC_MIXED, rel_tol=1e-12)
    po, do, _ = O.predict_solves(inp, opts)
    pg, dg, st = PR.PredictSolves(I, J, K)(inp, opts)
    for c in range(3):
        assert np.array_equal(dg[c], do[c])
        assert np.abs(pg[c] - po[c]).max() <= 1e-9 * np.abs(po[c]).max()


@pytest.mark.parametrize("I,J,K", BOXES[1:])
def test_geometry_segments(gpu_lib, I, J, K):
    """Face segments of 4, 8 and 16 cells; numbering columns with remainders."""
    g = GM.geometry_inputs("box", shape=(I, J, K), solid=W.SPHERE_C1)
    ref = O.grid_preprocess(g)
    got = g.copy()
    GM.GridPreprocess(I, J, K)(got)
    for f in GM.FAMILIES:
        assert got.fams[f].ext_cell == ref.fams[f].ext_cell
        for k in GM.OUTPUTS:
            a, b = got.fams[f].arrays.get(k), ref.fams[f].arrays.get(k)
            assert (a is None and b is None) or a.tobytes(order="F") == b.tobytes(order="F"), (f, k)
