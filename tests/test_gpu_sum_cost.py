"""The cost of a BiCGStab sum over the blocks of a 256^3 grid (8192), where a launch
of its own forms it: a second sum from the same partials adds at most what the
first one takes."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_second_sum_costs_no_more_than_the_first(gpu_lib, tmp_path):
    from simcoflow3d_gb300 import build as B
    lib = os.path.join(str(tmp_path), "sum_cost.so")
    r = subprocess.run([B.nvcc(), "-O3", "-std=c++17", "-shared", *B.ARCH, "-Xcompiler", "-fPIC",
                        "--expt-relaxed-constexpr", "-I" + B.CSRC, os.path.join(HERE, "sum_cost.cu"), "-o", lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    us = (C.c_float * 3)()
    assert C.CDLL(lib).sum_cost(8192, us) == 0
    print([round(v, 2) for v in us])
    assert us[1] < 2 * us[0] and us[2] < 2 * us[0], list(us)
