"""The quotients of the split-statistics and distance passes (pair_quotients)
and of the running means and shares (markstein_q) as compiled for the device,
bit for bit the correctly rounded division's over the callers' ranges."""

import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("quotients") / "libquotients.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode=arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-Xcompiler",
                    "-fPIC", "-shared", "-I" + os.path.join(ROOT, "openpgl_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "quotient_check.cu"), "-o", out], check=True)
    dll = ctypes.CDLL(out)
    dll.quotient_check.restype = ctypes.c_longlong
    return dll


@pytest.mark.parametrize("mode", range(6), ids=["denormal", "halfway", "small", "ordinary", "zero", "markstein"])
def test_quotients_are_the_divisions(lib, mode):
    assert lib.quotient_check(ctypes.c_uint64(1 << 26), mode) == 0
