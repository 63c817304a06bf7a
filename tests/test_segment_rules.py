"""Cells per column segment of the geometry's face kernel, by the grid.  CPU only."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    from simcoflow3d_gb300 import build as B
    try:
        nvcc = B.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    lib = str(tmp_path_factory.mktemp("rules") / "rules.so")
    r = subprocess.run([nvcc, "-std=c++17", "-shared", *B.ARCH, "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
                        "-I" + B.CSRC, os.path.join(HERE, "segment_rules.cu"), "-o", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(lib).geometry_segment


# flat grids whose columns give two blocks to each SM: segments of two took a
# tenth to a fifth longer than one segment
@pytest.mark.parametrize("box,cells", [((200, 200, 8), 4), ((220, 220, 8), 4), ((240, 160, 8), 4), ((256, 180, 8), 4),
                                       ((256, 180, 7), 4)])
def test_flat_grids_keep_segments_of_four(rule, box, cells):
    assert rule(*box) == cells


@pytest.mark.parametrize("box,cells", [((96, 96, 96), 4), ((64, 64, 64), 2), ((96, 96, 40), 2), ((256, 256, 4), 2),
                                       ((300, 150, 6), 2), ((180, 180, 8), 2), ((320, 100, 9), 2), ((128, 128, 128), 16),
                                       ((256, 256, 256), 32), ((300, 300, 16), 8)])
def test_other_grids(rule, box, cells):
    assert rule(*box) == cells
