"""pair_quotients (pgl_math.cuh), the quotients of the split-statistics and
distance passes, built for the host with the library's flags: numerators
down to the smallest denormal, whose quotients are scaled and rounded back,
quotients half way between two denormals among them, must be the division's,
bit for bit.  Host code only."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SOURCE = """
#include "pgl_math.cuh"
extern "C" void quotients(const float *a, const float *b, long n, float *q) {
  using namespace pgl;
  for (long i = 0; i + 1 < n; i += 2) {
    float2 up, down;
    up.x = fabsf(a[i]) < kSmallNumerator ? 0x1p50f : 1.0f;
    up.y = fabsf(a[i + 1]) < kSmallNumerator ? 0x1p50f : 1.0f;
    down = float2{1.0f / up.x, 1.0f / up.y};
    const float2 r = pair_quotients(float2{a[i], a[i + 1]}, float2{b[i], b[i + 1]},
                                    float2{1.0f / b[i], 1.0f / b[i + 1]}, up, down);
    q[i] = r.x;
    q[i + 1] = r.y;
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


@pytest.mark.parametrize("what", ["denormal_quotients", "halfway", "small", "ordinary", "zero"])
def test_quotients_are_the_divisions(lib, what):
    rng = np.random.default_rng(5)
    n = 2_000_000
    if what == "denormal_quotients":
        a, b = _floats(rng, n, 0, 40), np.abs(_floats(rng, n, 110, 140))
    elif what == "halfway":  # a = (m + 1/2) 2^-149 b for small integers b, most of them representable
        b = rng.integers(1, 4096, n).astype(np.float32)
        half = (2 * rng.integers(0, 4096, n) + 1).astype(np.float64) * 2.0 ** -150
        a = (half * b).astype(np.float32)
    elif what == "small":  # up to 1e-10 over the divisors' whole range, [1e-20, 1e8]
        a, b = _floats(rng, n, 0, 93), np.abs(_floats(rng, n, 61, 152))
    elif what == "ordinary":  # 1e-10 and more
        a, b = _floats(rng, n, 94, 180), np.abs(_floats(rng, n, 61, 152))
    else:
        a, b = np.zeros(n, np.float32), np.abs(_floats(rng, n, 61, 152))
    q = np.zeros(n, np.float32)
    lib.quotients(a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(n),
                  q.ctypes.data_as(ctypes.c_void_p))
    with np.errstate(all="ignore"):
        r = a / b
    bad = q.view(np.uint32) != r.view(np.uint32)
    i = np.flatnonzero(bad)[:3]
    assert not bad.any(), (int(bad.sum()), a[i], b[i], q[i], r[i])
