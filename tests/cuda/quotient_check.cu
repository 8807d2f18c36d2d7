// pair_quotients and markstein_q (pgl_math.cuh) as the kernels use them, with the
// packed instructions and reciprocals from rcp_newton, against the correctly
// rounded division on hashed operand pairs; returns the number of differences.
#include <cuda_runtime.h>

#include <cstdint>

#include "pgl_math.cuh"

using namespace pgl;

__device__ uint32_t mix(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdULL;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ULL;
  x ^= x >> 33;
  return uint32_t(x);
}
// a random float with a biased exponent of [lo, hi] (0: denormals)
__device__ float pick(uint64_t key, uint32_t lo, uint32_t hi, bool sign) {
  const uint32_t h = mix(key);
  return __uint_as_float((sign ? h & 0x80000000u : 0u) | (lo + mix(key * 3 + 1) % (hi - lo + 1)) << 23 | (h & 0x7FFFFFu));
}
// mode 0: denormal quotients, 1: quotients half way between denormals, 2: numerators up to
// 1e-10, 3: larger ones, 4: zeros; 5: markstein_q where |a| and |a / b| lie in [1e-30, 1e30]
__device__ void operands(int mode, uint64_t key, float &a, float &b) {
  b = pick(key * 7 + 5, 61, 152, false);
  if (mode == 0) {
    a = pick(key, 0, 40, true);
    b = pick(key * 7 + 5, 110, 140, false);
  } else if (mode == 1) {
    b = float(1 + mix(key * 7 + 5) % 4095u);
    a = float(double(2u * (mix(key) % 4096u) + 1u) * 0x1p-150 * double(b));
  } else if (mode == 2) {
    a = pick(key, 0, 93, true);
  } else if (mode == 3) {
    a = pick(key, 94, 180, true);
  } else if (mode == 4) {
    a = 0.0f;
  } else {
    a = pick(key, 28, 226, true);
    b = pick(key * 7 + 5, 28, 226, true);
  }
}
__global__ void quotient_kernel(uint64_t n, int mode, unsigned long long *bad) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    float a[2], b[2], q[2];
    operands(mode, 2 * i * 0x9E3779B97F4A7C15ULL + 1, a[0], b[0]);
    operands(mode, (2 * i + 1) * 0x9E3779B97F4A7C15ULL + 1, a[1], b[1]);
    const float2 y = make_float2(rcp_newton(b[0]), rcp_newton(b[1]));
    if (mode < 5) {
      const bool s0 = fabsf(a[0]) < kSmallNumerator, s1 = fabsf(a[1]) < kSmallNumerator;
      const float2 r = pair_quotients(make_float2(a[0], a[1]), make_float2(b[0], b[1]), y,
                                      make_float2(s0 ? 0x1p50f : 1.0f, s1 ? 0x1p50f : 1.0f),
                                      make_float2(s0 ? 0x1p-50f : 1.0f, s1 ? 0x1p-50f : 1.0f));
      q[0] = r.x;
      q[1] = r.y;
    } else {
      q[0] = markstein_q(a[0], b[0], y.x);
      q[1] = markstein_q(a[1], b[1], y.y);
    }
    for (int k = 0; k < 2; ++k) {
      const float want = __fdiv_rn(a[k], b[k]);
      if (mode == 5) {
        const bool in = fabsf(a[k]) >= 1e-30f && fabsf(a[k]) <= 1e30f && fabsf(b[k]) >= 1e-30f && fabsf(b[k]) <= 1e30f &&
                        fabsf(want) >= 1e-30f && fabsf(want) <= 1e30f;
        if (!in) continue;
      }
      if (__float_as_uint(q[k]) != __float_as_uint(want)) atomicAdd(bad, 1ULL);
    }
  }
}

extern "C" long long quotient_check(uint64_t n, int mode) {
  unsigned long long *d = nullptr, h = 0;
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(h));
  quotient_kernel<<<1216, 256>>>(n, mode, d);
  const cudaError_t err = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return err == cudaSuccess ? (long long)(h) : -1;
}
