// rcp_newton (pgl_math.cuh) against 1 / b rounded to nearest for every mantissa
// of the octave 2^e <= b < 2^(e + 1); returns the number of differences.
#include <cuda_runtime.h>

#include <cstdint>

#include "pgl_math.cuh"

__global__ void rcp_check_kernel(int e, unsigned *bad) {
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 23); m += gridDim.x * blockDim.x) {
    const float b = __uint_as_float((uint32_t(e + 127) << 23) | m);
    if (__float_as_uint(pgl::rcp_newton(b)) != __float_as_uint(__fdiv_rn(1.0f, b))) atomicAdd(bad, 1u);
  }
}

extern "C" int rcp_check(int e) {
  unsigned *d = nullptr, h = 0;
  if (cudaMalloc(&d, sizeof(unsigned)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(unsigned));
  rcp_check_kernel<<<304, 256>>>(e, d);
  const cudaError_t err = cudaMemcpy(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return err == cudaSuccess ? int(h) : -1;
}
