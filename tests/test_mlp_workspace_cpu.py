"""The network entries' workspace against a CUDA runtime on the host (fake_cudart.cpp): what a call, a failure, a
thread's end and a device change leave allocated, and what is used after its context has ended.  Kernels do not run.
"""
import ctypes as C
import os
import shutil
import subprocess
import threading
import time

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fluidized_bed_master_b200", "csrc")
OK, E_CUDA = 0, -2
pytestmark = pytest.mark.skipif(not shutil.which("nvcc"), reason="needs nvcc")


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("mlp") / "libmlp_host.so")
    subprocess.run(["nvcc", "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                    "--expt-extended-lambda", "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-o", so, os.path.join(CSRC, "mlp.cu"),
                    os.path.join(HERE, "fake_cudart.cpp")], check=True)
    lib = C.CDLL(so)
    lib.sphdem_mlp_forward.argtypes = [C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    return lib


def _forward(L):
    n = L.sphdem_mlp_param_count()
    feat, par, out = (C.c_uint16 * 160)(), (C.c_float * n)(), (C.c_float * 10)()
    return L.sphdem_mlp_forward(C.addressof(feat), 10, C.addressof(par), C.addressof(out), None)


def _in_thread(L, f):
    """f() in a thread of its own, whose end frees its workspace (join returns a moment earlier)."""
    err = []

    def run():
        try:
            f()
        except BaseException as e:   # noqa: BLE001  handed to the caller
            err.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    for _ in range(500):
        if not L.fake_live(0) and not L.fake_live(1):
            break
        time.sleep(0.01)
    if err:
        raise err[0]


def test_failed_kernel_attribute_leaves_nothing(L):
    def run():
        L.fake_fail_attribute(1)
        try:
            assert [_forward(L) for _ in range(3)] == [E_CUDA] * 3
            assert L.fake_live(0) == 0
        finally:
            L.fake_fail_attribute(0)
        assert _forward(L) == OK and L.fake_live(0) > 0

    _in_thread(L, run)
    assert L.fake_live(0) == 0 and L.fake_errors() == 0


def test_device_reset_ends_the_workspace(L):
    """The next call on the thread builds a new set, a thread's end after a reset frees nothing; neither uses what
    ended with the context."""
    def run():
        assert _forward(L) == OK
        n = L.fake_live(0)
        assert _forward(L) == OK and L.fake_live(0) == n > 0
        L.fake_reset()
        assert L.fake_live(0) == 0
        assert _forward(L) == OK and L.fake_live(0) == n and L.fake_errors() == 0
        L.fake_reset()

    _in_thread(L, run)
    assert L.fake_live(0) == 0 and L.fake_errors() == 0


def test_other_device_and_threads(L):
    def run():
        L.fake_device(0)
        assert _forward(L) == OK
        n = L.fake_live(0)
        L.fake_device(1)
        assert _forward(L) == OK and (L.fake_live(0), L.fake_live(1)) == (0, n)

        def inner():
            L.fake_device(0)
            assert _forward(L) == OK and (L.fake_live(0), L.fake_live(1)) == (n, n)

        t = threading.Thread(target=inner)
        t.start()
        t.join()
        for _ in range(500):
            if not L.fake_live(0):
                break
            time.sleep(0.01)
        assert (L.fake_live(0), L.fake_live(1)) == (0, n)

    _in_thread(L, run)
    assert L.fake_live(0) == L.fake_live(1) == 0 and L.fake_errors() == 0
