"""FP32 bounds of the redistancing's band distances: wherever FP32 decides
every branch, the FP64 distance lies inside the bounds (so a pair that the
bounds exclude cannot hold a target's minimum), and it decides most pairs."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    out = str(tmp_path_factory.mktemp("band_bounds") / "libband_bounds.so")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                        "-I" + os.path.join(HERE, "..", "simcoflow3d_gb300", "csrc"),
                        os.path.join(HERE, "band_bounds.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


@pytest.mark.parametrize("mode,decided", [(0, 0.9), (1, 0.4), (2, 0.5), (3, 0.0)])
@pytest.mark.parametrize("seed", [1, 2])
def test_distance_inside_its_bounds(lib, mode, decided, seed):
    out = (C.c_long * 4)()
    lib.check_bounds(C.c_uint(seed), C.c_long(4000), mode, out)
    pairs, bounded, bad, wide = list(out)
    assert pairs > 1000000 and bad == 0
    assert bounded >= decided * pairs


def test_one_face_equals_the_loop_over_axes(lib):
    """The nearest point on the face that outweighs the others, against the
    reference's loop over all three axes; ties take that loop."""
    lib.compare_faces.restype = C.c_long
    third = C.c_long()
    assert lib.compare_faces(C.c_uint(9), C.c_long(4000), C.byref(third)) == 0
    assert third.value > 1000000
