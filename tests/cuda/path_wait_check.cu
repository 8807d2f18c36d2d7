// Runs the path-sample kernel with a limit of its own on the looks for earlier
// tiles' counts, and with the first tiles left out (nobody takes them, so the
// waits for their counts run out).
#include <cstring>

#include "path_kernels.cu"

namespace pgl {
void count_launch() {}
}  // namespace pgl
using namespace pgl;

extern "C" int path_wait_check(const void *seg, size_t numSegments, const uint32_t *begin, uint32_t numPaths,
                               float maxDistance, uint32_t waitLimit, int tilesLeftOut, void *samples,
                               uint32_t *offsets) {
  char *d = nullptr;
  const size_t segBytes = numSegments * sizeof(PathSegmentRecord), beginBytes = (size_t(numPaths) + 1) * 4;
  const size_t outBytes = numSegments * sizeof(PGLSampleRecord), counts = path_counts_bytes(numPaths);
  const auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
  const size_t atBegin = up(segBytes), atOut = atBegin + up(beginBytes), atOffsets = atOut + up(outBytes),
               atCounts = atOffsets + up(beginBytes);
  if (cudaMalloc(&d, atCounts + counts) != cudaSuccess) return 1;
  int device = 0, sms = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaMemcpy(d, seg, segBytes, cudaMemcpyHostToDevice);
  cudaMemcpy(d + atBegin, begin, beginBytes, cudaMemcpyHostToDevice);
  cudaMemset(d + atOut, 0, outBytes);
  const auto *s = reinterpret_cast<const PathSegmentRecord *>(d);
  auto *o = reinterpret_cast<PGLSampleRecord *>(d + atOut);
  auto *b = reinterpret_cast<uint32_t *>(d + atBegin), *f = reinterpret_cast<uint32_t *>(d + atOffsets);
  const PathFlags fl{false, true, true};
  cudaError_t e = launch_path_samples(s, b, numPaths, maxDistance, fl, o, f, d + atCounts, sms, 0, waitLimit);
  if (e == cudaSuccess && tilesLeftOut > 0) {  // once more, without its first tiles
    const unsigned long long ticket = (unsigned long long)tilesLeftOut;
    e = cudaDeviceSynchronize();
    cudaMemset(d + atCounts, 0, counts);
    cudaMemcpy(d + atCounts, &ticket, sizeof(ticket), cudaMemcpyHostToDevice);
    cudaMemset(f, 0, beginBytes);
    const uint32_t most = most_tiles(numPaths), blocks = uint32_t(kPathBlocksPerSM * sms);
    path_samples_kernel<<<most < blocks ? most : blocks, kPathThreads, sizeof(PathShared)>>>(
        s, b, numPaths, maxDistance, fl, d + atCounts, waitLimit, f, o);
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  cudaMemcpy(samples, o, outBytes, cudaMemcpyDeviceToHost);
  cudaMemcpy(offsets, f, beginBytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}
