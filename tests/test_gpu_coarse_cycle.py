"""The V-cycle's small levels in one launch (csrc/k_coarse.cu) against the
oracle's CPU V-cycle, where that kernel's shares and paths end: levels of
exactly, and one column over, what the cluster takes (8192 cells of a point
level) and what one block owns (512 cells; 128 in FP64), partial line
segments, the smallest and largest degree.  FP64 V-cycle to 1e-12, FP32 to
2e-5 (relative L2): rounding of some ten thousand operations of 1e-16, and of
6e-8, as for the one-level kernels.  Thin boxes coarsen some levels in one or
two directions only, which the oracle's hierarchy weighs differently: there
the V-cycle is held to its symmetry, (M r, s) = (r, M s), to the same bounds."""
import numpy as np
import pytest

from simcoflow3d_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(32, 16, 16), (33, 16, 16), (8, 8, 8), (9, 8, 8), (8, 4, 4), (36, 30, 62)]
THIN = [(3, 4, 61), (150, 3, 5), (64, 64, 2)]


@pytest.mark.parametrize("degree", [1, 2, 8])
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 2e-5)])
@pytest.mark.parametrize("lines", [0, 1])
@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("shape", SHAPES + THIN)
def test_small_levels_match_oracle(gpu_lib, shape, walls, lines, precision, tol, degree):
    from oracle import oracle as O
    from simcoflow3d_gb300.projection import Projection
    w = W.build_workload("coarse-cycle", *shape, liquid=("bubble", 0.5, 0.5, 0.6, 0.2), rho_l=1000.0, rho_g=1.2,
                         extent=tuple((0.0, n / 32.0) for n in shape), bcp_flag=(1, 1, 1, 1, 1, int(walls)))
    p = Projection.for_workload(w, rel_tol=1e-6, precision=precision, smoother_degree=degree, smoother_lines=lines)
    pc, _, _ = p.poisson_solve(w)
    act = np.zeros(w.shape_g, dtype=bool)
    act[1:-1, 1:-1, 1:-1] = w.arrays["cell_type"] != 2
    rng = np.random.default_rng(23)

    def residual():
        r = np.where(act, rng.normal(size=w.shape_g), 0.0)
        if all(f == 1 for f in w.bcp_flag):
            r[act] -= r[act].mean()
        return np.asfortranarray(r)

    r = residual()
    z = p.debug_precondition(r)
    if shape in THIN:
        s = residual()
        y = p.debug_precondition(s)
        assert abs(np.vdot(z, s) - np.vdot(r, y)) <= tol * np.linalg.norm(z) * np.linalg.norm(s)
    else:
        zr = O.gmg_vcycle(w, pc, r, precision=0, degree=degree, line_seg=8 if lines else 0)
        err = np.linalg.norm(z - zr) / np.linalg.norm(zr)
        assert err <= tol, err
    assert not z[~act].any()
    p.close()
