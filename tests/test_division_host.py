"""div_rcp_try (pgl_math.cuh), the quotient of the split-statistics and
distance passes, built for the host with the library's flags: numerators
down to the smallest denormal, whose quotients are scaled and rounded back,
quotients half way between two denormals among them, against the division.
Where it reports a quotient it must be the division's, bit for bit; what it
may leave to the division is checked too.  Host code only."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SOURCE = """
#include "pgl_math.cuh"
extern "C" void quotients(const float *a, const float *b, long n, float *q, unsigned char *ok) {
  for (long i = 0; i < n; ++i) {
    bool k = true;
    q[i] = pgl::div_rcp_try(a[i], b[i], pgl::rcp_for_div(b[i]), k);
    ok[i] = k;
  }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    (d / "q.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math",
                    "-I" + os.path.join(ROOT, "openpgl_gb300", "csrc"), "-I" + CUDA_INCLUDE, str(d / "q.cpp"), "-o",
                    str(d / "q.so")], check=True)
    return ctypes.CDLL(str(d / "q.so"))


def _floats(rng, n, lo, hi):
    """Random floats of either sign with biased exponents in [lo, hi] (0: denormals)."""
    e = rng.integers(lo, hi + 1, n, dtype=np.uint32)
    return ((rng.integers(0, 2, n, dtype=np.uint32) << 31) | (e << 23)
            | rng.integers(0, 1 << 23, n, dtype=np.uint32)).view(np.float32)


@pytest.mark.parametrize("what", ["denormal_quotients", "halfway", "any", "zeros_and_edges"])
def test_quotients_are_the_divisions(lib, what):
    rng = np.random.default_rng(5)
    n = 2_000_000
    must = None
    if what == "denormal_quotients":
        a, b = _floats(rng, n, 0, 40), _floats(rng, n, 110, 140)
        must = True
    elif what == "halfway":  # a = (m + 1/2) 2^-149 b for small integers b, most of them representable
        b = rng.integers(1, 4096, n).astype(np.float32)
        half = (2 * rng.integers(0, 4096, n) + 1).astype(np.float64) * 2.0 ** -150
        a = (half * b).astype(np.float32)
        must = True
    elif what == "any":
        a, b = _floats(rng, n, 0, 254), _floats(rng, n, 30, 224)
    else:
        edge = np.array([0.0, -0.0, 1e-45, -1e-45, 1.1754944e-38, 1e-10, 9.9999994e-11, 1e30, 1.1e30, 3e38, np.inf,
                         -np.inf, np.nan, 1.0, -1.0], np.float32)
        a, b = (v.reshape(-1).copy() for v in np.meshgrid(edge, edge[2:]))
    q, ok = np.zeros(len(a), np.float32), np.zeros(len(a), np.uint8)
    lib.quotients(a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(len(a)),
                  q.ctypes.data_as(ctypes.c_void_p), ok.ctypes.data_as(ctypes.c_void_p))
    with np.errstate(all="ignore"):
        r = a / b
    bad = (ok == 1) & (q.view(np.uint32) != r.view(np.uint32)) & ~(np.isnan(q) & np.isnan(r))
    i = np.flatnonzero(bad)[:3]
    assert not bad.any(), (a[i], b[i], q[i], r[i])
    if must:
        assert (ok == 1).all()
    # out of range: always left to the division
    out = ~(np.abs(b) >= np.float32(1e-30)) | ~(np.abs(b) <= np.float32(1e30)) | ~(np.abs(a) <= np.float32(1e30))
    assert not ok[out].any()
