"""The transport's sweeps with shared faces and quotients against the general
sweep, bit for bit: every axis and stage, spacings that are powers of two,
uniform, different in every cell, repeating and tiny, and fields with signed
zeros, infinities and NaN; the quotients against the division; and the
interval that replaces the normals' gradient test."""
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
    out = str(tmp_path_factory.mktemp("sweep_lines") / "libsweep_lines.so")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                        "-I" + os.path.join(HERE, "..", "simcoflow3d_gb300", "csrc"),
                        os.path.join(HERE, "sweep_lines.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    L.compare_lines.restype = L.compare_quotients.restype = L.compare_gradient_test.restype = C.c_long
    return L


@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("values", [0, 1])
def test_lines_equal_general_sweep(lib, kind, values):
    for axis in range(3):
        for stage in range(3):
            for shape in ((9, 8, 7), (3, 5, 4), (4, 3, 3)):
                bad = lib.compare_lines(C.c_uint(17 * axis + stage + 100 * kind), *shape, axis, stage, kind, values)
                assert bad == 0, (axis, stage, shape, bad)


def test_quotients_equal_division(lib):
    assert lib.compare_quotients(C.c_uint(3), C.c_long(4000000)) == 0


def test_gradient_interval_equals_the_square_root_test(lib):
    assert lib.compare_gradient_test(C.c_uint(5), C.c_long(400000)) == 0
