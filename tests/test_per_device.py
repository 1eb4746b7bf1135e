"""Kernel attributes and the number of SMs are kept per device: a second device of the
process gets its own, a failure is tried again, and several threads may ask at once."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("dev") / "dev.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-shared", "-fPIC", "-pthread",
                        "-I", os.path.join(ROOT, "xbeach_gpu_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cxx", "per_device.cpp"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(so)


def test_each_device_once(lib):
    assert lib.get(0, 7) == 7 and lib.get(0, 9) == 7 and lib.made(0) == 1
    assert lib.get(1, 9) == 9 and lib.get(1, 7) == 9 and lib.made(1) == 1
    assert lib.get(2, 0) == 0 and lib.get(2, 4) == 4 and lib.get(2, 5) == 4 and lib.made(2) == 2
    assert lib.get(70, 3) == 3 and lib.get(70, 4) == 4 and lib.made(70) == 2   # beyond the table: made every time
    assert lib.get(-1, 3) == 0


def test_threads(lib):
    assert lib.race(3, 8) == 8000 and 1 <= lib.made(3) <= 8


def test_launchers_keep_nothing_per_process():
    """No launcher of the tensor-core kernels sets an attribute behind a plain flag."""
    src = open(os.path.join(ROOT, "xbeach_gpu_b200", "csrc", "nn_gemm.cu")).read()
    assert "static bool" not in src and "static int sms" not in src
