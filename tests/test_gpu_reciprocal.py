"""rcp_newton, the reciprocals of the split-statistics and distance passes:
correctly rounded for every mantissa, over the exponents of [1e-30, 1e30]."""

import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rcp") / "librcp.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode=arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-Xcompiler",
                    "-fPIC", "-shared", "-I" + os.path.join(ROOT, "openpgl_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "rcp_check.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("exponents", [(-100, -1), (0, 24), (25, 99)])
def test_every_mantissa(lib, exponents):
    for e in range(exponents[0], exponents[1] + 1):
        assert lib.rcp_check(e) == 0, e
