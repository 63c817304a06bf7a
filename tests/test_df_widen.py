"""The double-float to FP64 conversion on the integer pipe gives the bits of
the FP64 addition for every kind of pair."""
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
    out = str(tmp_path_factory.mktemp("df_widen") / "libdf_widen.so")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                        "-I" + os.path.join(HERE, "..", "simcoflow3d_gb300", "csrc"),
                        os.path.join(HERE, "df_widen.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(out)
    lib.check_widen.restype = C.c_long
    return lib


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_widening_equals_the_addition(lib, mode):
    assert lib.check_widen(C.c_uint(7 + mode), C.c_long(4000000), mode) == 0
