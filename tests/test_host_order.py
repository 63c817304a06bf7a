"""What the library's host code leaves unfinished on the GPU when a call returns,
and the order in which it gives work to its streams, over a stand-in CUDA
runtime (fake_cuda.h).  CPU only."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "simcoflow3d_gb300", "csrc")


def build(tmp, name):
    from simcoflow3d_gb300 import build as B
    try:
        nvcc = B.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    lib = os.path.join(str(tmp), name + ".so")
    # only the calls that a path reaches are defined, so the rest is bound lazily
    cmd = [nvcc, "-O1", "-std=c++17", "-shared", "-cudart", "none", *B.ARCH, "--expt-relaxed-constexpr", "-Xcompiler",
           "-fPIC", "-I" + CSRC, "-I" + HERE, os.path.join(HERE, name + ".cu"), os.path.join(HERE, "fake_cuda.cpp"),
           "-o", lib, "-Xlinker", "-z", "-Xlinker", "lazy", "-Xlinker", "-Bsymbolic", "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lib


def run(lib, *args):
    """The words that the library's `scenario` prints, in a process of its own."""
    code = ("import ctypes as C, sys\n"
            "args = [a.encode() for a in sys.argv[2:]]\n"
            "dl = C.CDLL(None)\n"
            "dl.dlopen.restype = dl.dlsym.restype = C.c_void_p\n"
            "dl.dlsym.argtypes = [C.c_void_p, C.c_char_p]\n"
            "h = dl.dlopen(sys.argv[1].encode(), 1)\n"   # RTLD_LAZY
            "f = C.CFUNCTYPE(None, C.c_char_p)(dl.dlsym(h, b'scenario'))\n"
            "f(args[0] if args else b'')\n")
    r = subprocess.run([sys.executable, "-c", code, lib, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    return r.stdout.split()


def test_predictor_create_leaves_nothing_to_other_streams(tmp_path):
    """The counter that tells a pass's last block, and every other zeroed buffer,
    before any of the context's three streams can use it."""
    rc, left = run(build(tmp_path, "host_predictor"))
    assert rc == "0" and left == "0"


@pytest.fixture(scope="module")
def projection(tmp_path_factory):
    return build(tmp_path_factory.mktemp("host"), "host_projection")


def test_projection_buffers_are_zeroed_on_its_own_stream(projection):
    """Those made after the context (a new plan, the adjoint's) too: nothing is
    left to the legacy stream, which its streams do not order after."""
    assert run(projection, "replan") == ["0", "0", "0"]


@pytest.mark.parametrize("where", ["nonfinite_rhs", "nonfinite_step"])
def test_failed_solve_leaves_nothing_running(projection, where):
    """Calls are synchronous, also those that end in an error."""
    assert run(projection, where) == ["1", "0", "0"]


def test_hierarchy_waits_for_the_inverse_before_it(projection):
    """A zero right-hand side ends a solve with the coarsest inverse still
    reading the levels on its own stream."""
    assert run(projection, "zero_rhs") == ["0", "0", "1"]


def test_warm_start_reads_its_own_residual(projection):
    """The residual a warm start begins with goes to no slot that the host reads
    later: nothing fences its write against the one the host waits for."""
    assert run(projection, "warm") == ["0", "1", "0"]


@pytest.mark.parametrize("how,polls,yields,waits", [("spin", 1, 0, 0), ("yield", 1, 1, 0), ("block", 0, 0, 1)])
def test_waiting_follows_the_device_flags(projection, how, polls, yields, waits):
    """A caller that chose blocking or yielding synchronisation gets it."""
    assert run(projection, how) == ["0", str(polls), str(yields), str(waits)]


def test_transport_buffers_are_zeroed_on_its_own_stream(tmp_path):
    """A zero fill on the legacy stream could land on fields staged meanwhile."""
    assert run(build(tmp_path, "host_transport")) == ["0", "0"]
