// two_pi_times, div3, lib_sincosf_any (pgl_math.cuh) and dqt_phi (dqt.cuh) against
// what they stand for (the tables of the C library's exceptions empty); each
// returns the number of differences, or -1.
#include <cuda_runtime.h>

#include <cstdint>

#include "dqt.cuh"

// every float of [0, 2.5) against the double product rounded once
__global__ void two_pi_kernel(unsigned *bad) {
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < 0x40200000u; b += gridDim.x * blockDim.x) {
    const float u = __uint_as_float(b);
    if (__float_as_uint(pgl::two_pi_times(u)) != __float_as_uint(float(2.0 * 3.14159265358979323846 * double(u))))
      atomicAdd(bad, 1u);
  }
}
// every float of [0, 1.5) as a point's y; every float of (-8.5, 8.5) as an angle
__global__ void phi_kernel(unsigned *bad) {
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < 0x3fc00000u; b += gridDim.x * blockDim.x) {
    const float y = __uint_as_float(b);
    if (__float_as_uint(pgl::dqt_phi(y)) !=
        __float_as_uint(float((double(y) - 0.5) * 2.0 * 3.14159265358979323846)))
      atomicAdd(bad, 1u);
  }
}
__global__ void sincos_kernel(unsigned *bad) {
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < 0x41080000u; b += gridDim.x * blockDim.x)
    for (int sign = 0; sign < 2; ++sign) {
      const float x = sign ? -__uint_as_float(b) : __uint_as_float(b);
      float s, c;
      pgl::lib_sincosf_any(x, &s, &c);
      float want = float(sin(double(fabsf(x))));
      want = x < 0.0f ? -want : want;
      if (__float_as_uint(s) != __float_as_uint(want) || __float_as_uint(c) != __float_as_uint(float(cos(double(x)))))
        atomicAdd(bad, 1u);
    }
}
__device__ uint32_t hash(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu;
  return x ^ (x >> 16);
}
// n random vectors and divisors; mode 0: of ordinary size, 1: any bit patterns,
// 2: ordinary ones with components replaced by zeros, infinities, NaN, the
// smallest numbers and the edges of the fast range
__global__ void div3_kernel(uint32_t n, int mode, unsigned *bad) {
  const uint32_t special[16] = {0u, 0x80000000u, 0x7f800000u, 0xff800000u, 0x7fc00000u, 1u, 0x80000001u, 0x00800000u,
                                0x26901D7Cu, 0x26901D7Du, 0xA6901D7Du, 0x58635FA9u, 0x58635FAAu, 0xD8635FA9u,
                                0x3f800000u, 0x7f7fffffu};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t v[4];
    for (uint32_t k = 0; k < 4; ++k) {
      v[k] = hash(4 * i + k + 77);
      if (mode != 1) v[k] = (v[k] & 0x80ffffffu) | (0x38000000u + ((v[k] & 0x0f000000u) >> 1));  // 2^-15 .. 2^1
      const uint32_t r = hash(v[k] ^ 0x9e3779b9u);
      if (mode == 2 && (r & 3u) == 0u) v[k] = special[(r >> 8) & 15u];
    }
    const pgl::V3 a = pgl::mk(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]));
    const float b = mode == 1 || mode == 2 ? __uint_as_float(v[3]) : fabsf(__uint_as_float(v[3]));
    const pgl::V3 q = pgl::div3(a, b);
    const float want[3] = {__fdiv_rn(a.x, b), __fdiv_rn(a.y, b), __fdiv_rn(a.z, b)}, got[3] = {q.x, q.y, q.z};
    for (int k = 0; k < 3; ++k)
      if (__float_as_uint(want[k]) != __float_as_uint(got[k]) && !(want[k] != want[k] && got[k] != got[k]))
        atomicAdd(bad, 1u);
  }
}

static int count(cudaError_t launched, unsigned *d) {
  unsigned h = 0;
  const cudaError_t err = cudaMemcpy(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return launched == cudaSuccess && err == cudaSuccess ? int(h) : -1;
}
extern "C" int two_pi_check() {
  unsigned *d = nullptr;
  if (cudaMalloc(&d, sizeof(unsigned)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(unsigned));
  two_pi_kernel<<<1216, 256>>>(d);
  return count(cudaGetLastError(), d);
}
extern "C" int phi_check() {
  unsigned *d = nullptr;
  if (cudaMalloc(&d, sizeof(unsigned)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(unsigned));
  phi_kernel<<<1216, 256>>>(d);
  return count(cudaGetLastError(), d);
}
extern "C" int sincos_check() {
  unsigned *d = nullptr;
  if (cudaMalloc(&d, sizeof(unsigned)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(unsigned));
  sincos_kernel<<<1216, 256>>>(d);
  return count(cudaGetLastError(), d);
}
extern "C" int div3_check(unsigned n, int mode) {
  unsigned *d = nullptr;
  if (cudaMalloc(&d, sizeof(unsigned)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(unsigned));
  div3_kernel<<<1216, 256>>>(n, mode, d);
  return count(cudaGetLastError(), d);
}
