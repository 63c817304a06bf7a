"""The FP32 bounds of the redistancing's band distances in the arithmetic the GPU
forms them with: fused multiply-adds, and a square root off by as much as the
approximate one may be (2^-23 of its value), either way."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=["-0x1p-23", "0x1p-23"])
def lib(request, tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    out = str(tmp_path_factory.mktemp("band_arithmetic") / "libband.so")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                        "-DTR_SQRT_ERROR=" + request.param,
                        "-I" + os.path.join(HERE, "..", "simcoflow3d_gb300", "csrc"),
                        os.path.join(HERE, "band_arithmetic.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    L.host_fma.restype = L.host_sqrt.restype = C.c_float
    L.host_fma.argtypes = [C.c_float] * 3
    L.host_sqrt.argtypes = [C.c_float]
    return L, float.fromhex(request.param)


def test_the_host_build_has_the_gpus_operations(lib):
    L, err = lib
    a = 1.0 + 2.0 ** -12
    assert L.host_fma(a, a, -1.0) == 2.0 ** -11 + 2.0 ** -24   # the product is not rounded
    assert L.host_sqrt(2.25) == C.c_float(1.5 * (1.0 + err)).value   # rounded to FP32


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("seed", [3, 4])
def test_distance_inside_its_bounds(lib, mode, seed):
    """No bound is wider than 0.1 of the cell's scale for what a reconstruction
    gives: the error is at most 5e-4 a branch where a foot point is taken, and
    where a face's line is followed (slope up to 50) 3.1e-4 x 50 of the foot and
    2e-6 of an intercept and a distance below 50 x 126 each, 0.041 either way."""
    out = (C.c_long * 4)()
    lib[0].check_bounds(C.c_uint(seed), C.c_long(3000), mode, out)
    pairs, bounded, bad, wide = list(out)
    assert pairs > 1000000 and bad == 0
    if mode < 3:
        assert wide == 0
