"""Where the last block of an FP32 BiCGStab pass forms the grid's sums: only on
grids that are resident at once, since the sums' registers cost the passes
warps.  And the results at block counts on both sides of that limit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from simcoflow3d_gb300 import capi, geometry as GM, predictor as PR, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_summing_grids_are_resident_at_once(gpu_lib, tmp_path):
    from simcoflow3d_gb300 import build as B
    lib = os.path.join(str(tmp_path), "resident.so")
    r = subprocess.run([B.nvcc(), "-O3", "-std=c++17", "-shared", *B.ARCH, "-Xcompiler", "-fPIC",
                        "--expt-relaxed-constexpr", "-I" + B.CSRC, os.path.join(HERE, "resident_blocks.cu"), "-o", lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    resident, limit = (C.c_int * 3)(), (C.c_int * 3)()
    assert C.CDLL(lib).resident_blocks(resident, limit) == 0
    assert all(m <= n for m, n in zip(limit, resident)), (list(limit), list(resident))


# 1350 and 2700 blocks: FP32 P and S sum in their last block and in a launch;
# FP64 the same at 2430 and 2439
@pytest.mark.parametrize("precision,J", [(capi.SCF_PREC_MIXED, 600), (capi.SCF_PREC_MIXED, 1200),
                                         (capi.SCF_PREC_FP64, 1080), (capi.SCF_PREC_FP64, 1084)])
def test_sums_beside_the_limit(gpu_lib, precision, J):
    """Dp bit for bit; the velocities of two solves to a residual of 1e-12 agree
    to 1e-12 times the systems' condition, a few hundred: 1e-9 (relative L2)."""
    I, K = 3, 129
    g = O.grid_preprocess(GM.geometry_inputs("box", shape=(I, J, K), solid=W.SPHERE_C1))
    inp = PR.momentum_inputs(g, vof_old_noise=0.01)
    opts = PR.default_opts(precision=precision, rel_tol=1e-12)
    po, do, _ = O.predict_solves(inp, opts)
    pg, dg, _ = PR.PredictSolves(I, J, K)(inp, opts)
    for c in range(3):
        assert np.array_equal(dg[c], do[c])
        assert np.linalg.norm(pg[c] - po[c]) <= 1e-9 * np.linalg.norm(po[c])
