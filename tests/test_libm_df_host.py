"""The double-float exp and lobe normalisations of the merge costs
(pgl_math.cuh) built for the host: accuracy against long double, and every
result that their rounding test decides equal to the double-precision form
rounded once.  Host code only."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("libm") / "libmdf.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math",
                    "-I" + os.path.join(ROOT, "openpgl_gb300", "csrc"), "-I" + CUDA_INCLUDE,
                    os.path.join(ROOT, "tests", "cuda", "libm_df_host.cpp"), "-o", out], check=True)
    dll = ctypes.CDLL(out)
    dll.expf_df_check.argtypes = [ctypes.c_uint32] * 3 + [ctypes.c_float] + [ctypes.c_void_p] * 2
    dll.norms_df_check.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_long, ctypes.c_void_p]
    return dll


def _bits(f):
    return int(np.float32(f).view(np.uint32))


@pytest.mark.parametrize("lo,hi,decided", [(0.0, 90.0, 0.99), (-0.0, -87.0, 0.99), (-87.0, -104.0, 0.0),
                                           (-104.1, -4e5, 1.0), (1e-45, 1e-30, 1.0)])
@pytest.mark.parametrize("margin", [0.0, 2.0 ** -33])
def test_exp(lib, lo, hi, decided, margin):
    out, err = np.zeros(3, np.uint64), np.zeros(1)
    lib.expf_df_check(_bits(lo), _bits(hi), 211, margin, out.ctypes.data, err.ctypes.data)
    n, undecided, wrong = (int(v) for v in out)
    assert n > 10000 and wrong == 0
    # the test widens by 2^-38; a result lies within w (relative) of a rounding
    # boundary on about 2^25 w of the inputs at most
    assert err[0] < 2.0 ** -40
    assert undecided <= (1 - decided + 2.0 ** 25 * (2.0 ** -38 + margin) * 1.5) * n


def test_normalisations(lib):
    rng = np.random.default_rng(3)
    n = 2_000_000
    k = np.exp(rng.uniform(np.log(1e-3), np.log(6.4e5), n)).astype(np.float32)
    e = np.exp(-2.0 * k.astype(np.float64)).astype(np.float32)
    e[::3] = rng.random((n + 2) // 3).astype(np.float32)
    e[:4], k[4:8] = (1.0, 0.0, 0.99999994, 1e-40), (0.0, np.inf, np.nan, 1e-20)
    s = np.exp(rng.uniform(-60, 60, n)).astype(np.float32)
    out = np.zeros(3, np.uint64)
    lib.norms_df_check(k.ctypes.data, e.ctypes.data, s.ctypes.data, n, out.ctypes.data)
    total, undecided, wrong = (int(v) for v in out)
    assert total == 2 * n and wrong == 0
    assert undecided < 0.5 * n  # a scale below 1e-15 or above 1e15, the edges put in above, and few others
