// Training samples from many paths' segments at once on the device
// (PathSegmentDataStorage.h:161-316 per path), in path order and, within a
// path, in the reference's order (last vertex first).
//
// One pass over the segments: a block stages the records of its paths in shared
// memory (they lie one after the other; a thread per path read 136-byte records
// a path apart), takes a thread per vertex, and learns where its samples go from
// the blocks before it (a decoupled look-back over per-block counts).
// 852,000 segments of 131,072 paths are 116 MB in and 17 MB out (19 us at the
// copy rate).  Two passes with a thread per path took 192 us, this one 77 us
// (paths of 1 to 24 segments 752 -> 246 us, of 1 or 2 25 -> 25 us): a tile stages
// for 5,500 cycles, prepares and deals out its vertices for 6,000, adds their
// contributions for 8,700 (bound by shared-memory reads, 15 words per step) and
// waits 6,900 for its place in the output.
#include <cuda_runtime.h>

#include "launch.h"
#include "path_samples.cuh"

namespace pgl {

constexpr int kPathThreads = 256, kPathWarps = kPathThreads / 32;
constexpr int kMaxTilePaths = 256, kMinTilePaths = 8;
constexpr int kStagedSegments = 480;  // 64 KB: three blocks per SM
constexpr int kTileSegments = 380;    // what a tile's paths have on average at most: a tile that has to be
                                      // staged in parts runs three times as long, and the tiles behind wait
constexpr int kPathRounds = (kStagedSegments + kPathThreads - 1) / kPathThreads;
constexpr int kPathBlocksPerSM = 3;
constexpr int kDepths = 64;  // bins of a tile's vertices by the segments behind them
constexpr int kRecordWords = sizeof(PathSegmentRecord) / 4;
static_assert(kRecordWords == 34 && sizeof(PGLSampleRecord) == 40, "staging works on the records' words");

// words of a staged record that carry results once their fields were read: the
// sample takes the first ten (position and directionIn are its own first six)
enum { kWeight = 6, kPdf = 7, kDistance = 8, kFlags = 9, kRcpRR = 31, kStep = 32, kFactor = 33 };
static_assert(offsetof(PathSegmentRecord, dox) == 4 * kWeight && offsetof(PathSegmentRecord, nx) == 4 * kFlags &&
                  offsetof(PathSegmentRecord, pad2) == 4 * kRcpRR && offsetof(PathSegmentRecord, regionPtr) == 4 * kStep,
              "words of results lie in fields that are no longer read, or never");

// where the paths of a tile lie
struct PathTile {
  uint32_t first;  // path
  int np;          // paths, 0 when there are no more tiles
  int apart;       // their records do not lie one after the other
  uint32_t tile;
  uint32_t pre[kMaxTilePaths + 1], items[kMaxTilePaths + 1];  // segments and vertices before each path
  uint32_t begin[kMaxTilePaths];
  __device__ __forceinline__ int n(int p) const { return int(pre[p + 1] - pre[p]); }
};
struct PathShared {
  PathTile tiles[2];  // this tile and the next
  uint32_t made[kPathRounds * kPathWarps], before[kPathRounds * kPathWarps + 1];
  uint32_t base, sorted;
  bool failed;
  uint32_t depth[kDepths];
  union {
    uint32_t order[kStagedSegments];  // vertices by depth: record, place in the path, the path's segments
    uint16_t vertexOf[kStagedSegments];
  };
  unsigned char madeAt[kStagedSegments];
  alignas(16) unsigned char stage[kStagedSegments * sizeof(PathSegmentRecord) + 16];
};
static_assert(kPathBlocksPerSM * (sizeof(PathShared) + 1024) <= 228 * 1024, "blocks per SM");

__device__ __forceinline__ PathShared &path_shared() {
  extern __shared__ __align__(16) unsigned char smem[];
  return *reinterpret_cast<PathShared *>(smem);
}

// distance of vertex i: from the next vertex that starts again (or the path's
// last) down, as the reference's loop from the path's end does
template <typename Step, typename Factor>
__device__ __forceinline__ float vertex_distance(int i, int n, float maxDistance, Step step, Factor factor) {
  int r = i + 1;
  while (r <= n - 2 && factor(r) != -1.0f) ++r;
  float last = 0.0f, distance = 0.0f;
  for (--r; r >= i; --r) {
    distance = fminf(step(r) + last, 2.0f * maxDistance);
    last = distance * (r > i ? factor(r) : 1.0f);
  }
  return distance;
}
// rr's reciprocal where div_by takes it
__device__ __forceinline__ float rr_reciprocal(float rr) { return rr >= 1e-12f && rr <= 1e12f ? rcp_newton(rr) : 0.0f; }

// The path of the tile that item x belongs to, among paths [a, z).
__device__ __forceinline__ int path_of(const PathTile &S, uint32_t x, int a, int z) {
  while (z - a > 1) {
    const int m = (a + z) >> 1;
    (S.items[m] <= x ? a : z) = m;
  }
  return a;
}
// exclusive prefix of the made counts, its total at the end
__device__ __forceinline__ uint32_t scan_made(PathShared &S) {
  __syncthreads();
  if (threadIdx.x < 32) {
    constexpr int kWords = kPathRounds * kPathWarps;
    static_assert(kWords <= 32, "a lane per word");
    const uint32_t v = threadIdx.x < kWords ? __popc(S.made[threadIdx.x]) : 0;
    uint32_t sum = v;
    for (int d = 1; d < 32; d *= 2) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, sum, d);
      if (int(threadIdx.x) >= d) sum += up;
    }
    if (threadIdx.x < kWords) S.before[threadIdx.x + 1] = sum;
    if (threadIdx.x == 0) S.before[0] = 0;
  }
  __syncthreads();
  return S.before[kPathRounds * kPathWarps];
}
__device__ __forceinline__ uint32_t made_before(const PathShared &S, uint32_t item) {
  const uint32_t w = item >> 5;
  if (w >= uint32_t(kPathRounds * kPathWarps)) return S.before[kPathRounds * kPathWarps];
  return S.before[w] + __popc(S.made[w] & ((1u << (item & 31)) - 1u));
}

// segment records of paths [a, z) (contiguous) into the stage; returns where
// the first one lies (16-byte copies where source and stage share the alignment)
__device__ __forceinline__ PathSegmentRecord *stage_segments(PathShared &S, const PathTile &T, const PathSegmentRecord *seg, int a,
                                                               int z) {
  const uint32_t count = T.pre[z] - T.pre[a];
  const unsigned char *src = reinterpret_cast<const unsigned char *>(seg + T.begin[a]);
  const uint32_t head = uint32_t(reinterpret_cast<uintptr_t>(src) & 15u);  // 0 or 8
  unsigned char *dst = S.stage + head;
  const uint32_t bytes = count * uint32_t(sizeof(PathSegmentRecord));
  const uint32_t lead = (16u - head) & 15u, body = bytes > lead ? (bytes - lead) / 16u : 0u;
  const uint32_t to = uint32_t(__cvta_generic_to_shared(dst));
  for (uint32_t i = threadIdx.x; i < body; i += kPathThreads)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + lead + 16u * i), "l"(src + lead + 16u * i));
  if (threadIdx.x == 0 && lead && bytes)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(src));
  if (threadIdx.x == 32 && bytes > lead && ((bytes - lead) & 15u))
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + bytes - 8u), "l"(src + bytes - 8u));
  asm volatile("cp.async.commit_group;");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  return reinterpret_cast<PathSegmentRecord *>(dst);
}

// The samples of the staged paths [a, z): made masks, vertexOf by rank, the
// samples in their vertices' words.  Returns their number.  A vertex's work is
// the segments behind it, so the vertices are dealt out by that number (a warp of
// neighbours would run as long as its deepest one: 2.7 times the work at paths
// of 1 to 12 segments), the deepest of the second half to the last threads.
__device__ __noinline__ uint32_t staged_samples(int buffer, const PathSegmentRecord *seg, int a, int z,
                                                float maxDistance, PathFlags fl) {
  PathShared &S = path_shared();
  const PathTile &T = S.tiles[buffer];
  const uint32_t items = T.items[z] - T.items[a];
  if (items == 0) {  // paths of one segment have no vertices: nothing to stage
    if (threadIdx.x == 0) S.before[0] = 0;
    __syncthreads();
    return 0;
  }
  if (threadIdx.x < kDepths) S.depth[threadIdx.x] = 0;
  PathSegmentRecord *stage = stage_segments(S, T, seg, a, z);
  float *words = reinterpret_cast<float *>(stage);
  int at[kPathRounds], bin[kPathRounds];
  uint32_t entry[kPathRounds], place[kPathRounds];
#pragma unroll
  for (int r = 0; r < kPathRounds; ++r) {
    const uint32_t x = uint32_t(r * kPathThreads) + threadIdx.x;
    at[r] = bin[r] = -1;
    if (x < items) {
      const int p = path_of(T, T.items[a] + x, a, z), n = T.n(p);
      const int vert = n - 2 - int(T.items[a] + x - T.items[p]);
      at[r] = int(T.pre[p] - T.pre[a]) + vert;
      const PathSegmentRecord &cur = stage[at[r]], &nxt = stage[at[r] + 1];
      words[at[r] * kRecordWords + kStep] = vertex_step(cur, nxt);
      words[at[r] * kRecordWords + kFactor] = vertex_factor(cur);
      words[(at[r] + 1) * kRecordWords + kRcpRR] = rr_reciprocal(nxt.rr);
      S.madeAt[at[r]] = 0;
      if (vertex_eligible(cur)) {
        bin[r] = max(kDepths - (n - 1 - vert), 0);
        place[r] = atomicAdd(&S.depth[bin[r]], 1u);
        entry[r] = uint32_t(at[r]) | uint32_t(vert) << 10 | uint32_t(n) << 20;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    static_assert(kDepths == 64 && kStagedSegments < 1024, "two bins per lane; ten bits per field of an entry");
    const uint32_t lo = S.depth[2 * threadIdx.x], hi = S.depth[2 * threadIdx.x + 1];
    uint32_t sum = lo + hi;
    for (int d = 1; d < 32; d *= 2) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, sum, d);
      if (int(threadIdx.x) >= d) sum += up;
    }
    S.depth[2 * threadIdx.x] = sum - lo - hi;
    S.depth[2 * threadIdx.x + 1] = sum - hi;
    if (threadIdx.x == 31) S.sorted = sum;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kPathRounds; ++r)
    if (bin[r] >= 0) S.order[S.depth[bin[r]] + place[r]] = entry[r];
  __syncthreads();
  const int sorted = int(S.sorted);
#pragma unroll 1
  for (int r = 0; r < kPathRounds; ++r) {
    const int k = r * kPathThreads + (r & 1 ? kPathThreads - 1 - int(threadIdx.x) : int(threadIdx.x));
    if (k >= sorted) continue;
    const uint32_t e = S.order[k];
    const int v = int(e & 1023u), vert = int(e >> 10 & 1023u), n = int(e >> 20);
    const PathSegmentRecord &cur = stage[v];
    const float *path = words + (v - vert) * kRecordWords;
    const float distance =
        vertex_distance(vert, n, maxDistance, [&](int i) { return path[i * kRecordWords + kStep]; },
                        [&](int i) { return path[i * kRecordWords + kFactor]; });
    float c[3];
    vertex_contribution(&cur, n - vert, fl,
                        [](const PathSegmentRecord &s) { return reinterpret_cast<const float *>(&s)[kRcpRR]; }, c);
    if (made_sample(c, distance)) {
      const float pdf = vertex_pdf(cur);
      const uint32_t flags = cur.volumeScatter ? 2u : 0u;  // EInsideVolume
      float *w = words + v * kRecordWords;
      w[kWeight] = sample_weight(c, pdf);
      w[kPdf] = pdf;
      w[kDistance] = distance;
      w[kFlags] = u2f(flags);
      S.madeAt[v] = 1;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kPathRounds; ++r) {
    const bool made = at[r] >= 0 && S.madeAt[at[r]] != 0;
    if (!made) at[r] = -1;
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, made);
    if ((threadIdx.x & 31) == 0) S.made[r * kPathWarps + (threadIdx.x >> 5)] = mask;
  }
  const uint32_t total = scan_made(S);
#pragma unroll
  for (int r = 0; r < kPathRounds; ++r)
    if (at[r] >= 0)
      S.vertexOf[made_before(S, uint32_t(r * kPathThreads) + threadIdx.x)] =
          uint16_t((at[r] * kRecordWords + int(words - reinterpret_cast<float *>(S.stage))) / 2);
  __syncthreads();
  return total;
}
// the staged samples of paths [a, z) to out[base ...], and where each path's begin
__device__ __forceinline__ void write_staged(const PathShared &S, const PathTile &T, int a, int z, uint32_t base,
                                             uint32_t total, uint32_t *offsets, PGLSampleRecord *out) {
  for (int p = a + int(threadIdx.x); p < z; p += kPathThreads)
    offsets[p] = base + made_before(S, T.items[p] - T.items[a]);
  const float *words = reinterpret_cast<const float *>(S.stage);
  float *to = reinterpret_cast<float *>(out + base);
  for (uint32_t x = threadIdx.x; x < total * 10u; x += kPathThreads) {
    const uint32_t rank = x / 10u;
    to[x] = words[2 * S.vertexOf[rank] + (x - 10u * rank)];
  }
  __syncthreads();  // the stage is free again
}

// A path with more segments than the stage holds: a thread per vertex on the
// records in memory; out == nullptr counts.  Its time grows with the square of the
// segments, so every thousand steps or so a thread says that it is still at it
// (any new value will do), and the tiles behind keep waiting.
__device__ __noinline__ uint32_t long_path(const PathSegmentRecord *seg, int n, float maxDistance,
                                           PathFlags fl, PGLSampleRecord *out, unsigned long long *progress) {
  PathShared &S = path_shared();
  uint32_t total = 0, steps = 0;
  const auto beat = [&] {
    if ((++steps & 1023u) == 0) *static_cast<volatile unsigned long long *>(progress) = (unsigned long long)clock64();
  };
  const auto step = [&](int v) { return vertex_step(seg[v], seg[v + 1]); };
  const auto factor = [&](int v) {
    beat();
    return vertex_factor(seg[v]);
  };
  const auto rcp = [&](const PathSegmentRecord &s) {
    beat();
    return rr_reciprocal(s.rr);
  };
  for (int top = n - 2; top >= 0; top -= kPathRounds * kPathThreads) {
    bool made[kPathRounds];
#pragma unroll 1
    for (int r = 0; r < kPathRounds; ++r) {
      const int i = top - (r * kPathThreads + int(threadIdx.x));
      made[r] = false;
      if (i >= 0 && vertex_eligible(seg[i])) {
        const float distance = vertex_distance(i, n, maxDistance, step, factor);
        float c[3];
        vertex_contribution(seg + i, n - i, fl, rcp, c);
        made[r] = made_sample(c, distance);
      }
      const uint32_t mask = __ballot_sync(0xFFFFFFFFu, made[r]);
      if ((threadIdx.x & 31) == 0) S.made[r * kPathWarps + (threadIdx.x >> 5)] = mask;
    }
    const uint32_t count = scan_made(S);
    if (out) {
#pragma unroll 1
      for (int r = 0; r < kPathRounds; ++r) {
        const int x = r * kPathThreads + int(threadIdx.x), i = top - x;
        if (!made[r]) continue;
        const PathSegmentRecord &cur = seg[i];
        float c[3];
        vertex_contribution(seg + i, n - i, fl, rcp, c);
        PGLSampleRecord o;
        o.px = cur.px;
        o.py = cur.py;
        o.pz = cur.pz;
        o.dx = cur.dix;
        o.dy = cur.diy;
        o.dz = cur.diz;
        o.pdf = vertex_pdf(cur);
        o.weight = sample_weight(c, o.pdf);
        o.distance = vertex_distance(i, n, maxDistance, step, factor);
        o.flags = cur.volumeScatter ? 2u : 0u;
        out[total + made_before(S, uint32_t(x))] = o;
      }
    }
    total += count;
    __syncthreads();
  }
  return total;
}

// The counts that say where a tile's samples go, in groups of 32 tiles.  All
// words start at zero: ticket, whether a wait ran out, the last sign of a long path
// at work, then per tile its samples (bit 63 set when known),
// per group the sum of its tiles' samples (the tiles added so far above bit 40)
// and the samples before it (bit 63 set when known).  A tile reads its group's
// tiles and up to 32 groups per step, so the blocks that wait at the same time
// do not crowd on a few lines (polling 128 tiles per step cost 22,000 cycles per
// tile, this 7,000).
constexpr unsigned long long kKnown = 1ull << 63;
constexpr int kGroupShift = 40;  // samples are fewer than 2^32: a group's sum stays below
struct TileCounts {
  unsigned long long *ticket, *failed, *progress, *tile, *group, *before;
  __host__ __device__ TileCounts(void *words, uint32_t numTiles) {
    const size_t groups = (size_t(numTiles) + 31) / 32;
    ticket = static_cast<unsigned long long *>(words);
    failed = ticket + 1;
    progress = ticket + 2;
    tile = ticket + 3;
    group = tile + numTiles;
    before = group + groups;
  }
  static size_t words(uint32_t numTiles) { return 3 + size_t(numTiles) + 2 * ((size_t(numTiles) + 31) / 32); }
};
__device__ __forceinline__ unsigned long long poll(const unsigned long long *p) {
  return *static_cast<const volatile unsigned long long *>(p);
}
// A wait's limit, in looks in vain (most of a microsecond each) since a long path last
// showed itself at work.  One wait that runs out fails the whole launch: every
// other wait ends too, and the total says so.
struct PathWait {
  uint32_t looks = 0;
  unsigned long long seen = 0;
  __device__ __forceinline__ bool over(const TileCounts &C, uint32_t limit) {
    if ((++looks & 63u) != 0) return false;  // many wait at once: they read the shared words now and then
    if (__shfl_sync(0xFFFFFFFFu, poll(C.failed), 0) != 0) return true;
    const unsigned long long now = __shfl_sync(0xFFFFFFFFu, poll(C.progress), 0);
    if (now != seen) {
      seen = now;
      looks = 0;
    }
    return looks >= limit;
  }
};
// Samples before this tile (one warp calls it).  Blocks take their tiles in
// order, each its next one only when this one's samples are counted, and wait
// for earlier tiles only, so the earliest tile not yet counted is always being
// worked on; the wait has a limit all the same.
__device__ __forceinline__ uint32_t samples_before(const TileCounts &C, uint32_t tile, uint32_t total, uint32_t limit,
                                                   bool *failed) {
  const int lane = threadIdx.x & 31;
  const uint32_t group = tile / 32, first = group * 32;
  if (lane == 0) {
    atomicExch(&C.tile[tile], kKnown | total);
    atomicAdd(&C.group[group], 1ull << kGroupShift | total);
  }
  PathWait wait;
  uint32_t sum = 0;
  for (int64_t last = int64_t(group) - 1; last >= 0;) {
    // groups last, last - 1, ...: their sums, down to one with the samples before it known
    const int64_t mine = last - lane;
    unsigned long long v = 32ull << kGroupShift, b = kKnown;
    if (mine >= 0) {
      v = poll(&C.group[mine]);
      b = mine > 0 ? poll(&C.before[mine]) : kKnown;
    }
    const unsigned full = __ballot_sync(0xFFFFFFFFu, (v >> kGroupShift) == 32);
    const unsigned known = __ballot_sync(0xFFFFFFFFu, (b & kKnown) != 0);
    const int stop = known ? __ffs(known) - 1 : 31;
    const unsigned need = 0xFFFFFFFFu >> (31 - stop);
    if ((full & need) == need) {
      sum += __reduce_add_sync(0xFFFFFFFFu, lane <= stop ? uint32_t(v) : 0u);
      if (known) {
        sum += __shfl_sync(0xFFFFFFFFu, uint32_t(b), stop);
        break;
      }
      last -= 32;
    } else {
      if ((*failed = wait.over(C, limit))) return 0;
      __nanosleep(200);
    }
  }
  if (tile == first && lane == 0) atomicExch(&C.before[group], kKnown | sum);
  for (;;) {
    const bool before = lane < int(tile - first);
    const unsigned long long v = before ? poll(&C.tile[first + lane]) : kKnown;
    if (__all_sync(0xFFFFFFFFu, (v & kKnown) != 0))
      return sum + __reduce_add_sync(0xFFFFFFFFu, before ? uint32_t(v) : 0u);
    if ((*failed = wait.over(C, limit))) return 0;
    __nanosleep(100);
  }
}

// One warp: the next tile's paths, their segments and vertices.
__device__ __forceinline__ void next_tile(PathTile &T, unsigned long long *ticket, uint32_t tiles, uint32_t perTile,
                                          const uint32_t *begin, uint32_t numPaths) {
  const int lane = threadIdx.x & 31;
  uint32_t tile = lane == 0 ? uint32_t(atomicAdd(ticket, 1ull)) : 0u;
  tile = __shfl_sync(0xFFFFFFFFu, tile, 0);
  const bool none = tile >= tiles;
  const uint32_t first = none ? numPaths : tile * perTile;
  const int np = int(min(perTile, numPaths - first));
  if (lane == 0) {
    T.tile = tile;
    T.first = first;
    T.np = np;
    T.pre[0] = T.items[0] = 0;
  }
  uint32_t sum = 0, vertices = 0;
  bool apart = false;
  for (int q = 0; q < np; q += 32) {
    const int p = q + lane;
    uint32_t b = 0;
    int n = 0;
    if (p < np) {
      b = begin[first + p];
      n = int(begin[first + p + 1] - b);
      T.begin[p] = b;
    }
    apart = apart || __any_sync(0xFFFFFFFFu, n < 0);
    n = n > 0 ? n : 0;
    uint32_t s = uint32_t(n), v = n > 1 ? uint32_t(n - 1) : 0u;
    for (int d = 1; d < 32; d *= 2) {
      const uint32_t us = __shfl_up_sync(0xFFFFFFFFu, s, d), uv = __shfl_up_sync(0xFFFFFFFFu, v, d);
      if (lane >= d) {
        s += us;
        v += uv;
      }
    }
    if (p < np) {
      T.pre[p + 1] = sum + s;
      T.items[p + 1] = vertices + v;
    }
    sum += __shfl_sync(0xFFFFFFFFu, s, 31);
    vertices += __shfl_sync(0xFFFFFFFFu, v, 31);
  }
  if (lane == 0) T.apart = apart;
}

__host__ __device__ inline uint32_t most_tiles(uint32_t numPaths) {
  return uint32_t((uint64_t(numPaths) + kMinTilePaths - 1) / kMinTilePaths);
}
__global__ void __launch_bounds__(kPathThreads, kPathBlocksPerSM)
path_samples_kernel(const PathSegmentRecord *seg, const uint32_t *begin, uint32_t numPaths, float maxDistance,
                    PathFlags fl, void *counts, uint32_t waitLimit, uint32_t *offsets, PGLSampleRecord *out) {
  PathShared &S = path_shared();
  const int warp = threadIdx.x >> 5;
  const TileCounts C(counts, most_tiles(numPaths));
  // paths per tile: what the stage holds of them on average (with few segments
  // per tile a block would wait more than work), fewer where that leaves blocks
  // without a tile
  const uint64_t segments = begin[numPaths] - begin[0];
  uint32_t perTile = kMaxTilePaths;
  if (perTile * segments > uint64_t(kTileSegments) * numPaths)
    perTile = max(uint32_t(uint64_t(kTileSegments) * numPaths / segments), uint32_t(kMinTilePaths));
  perTile = min(perTile, max((numPaths + gridDim.x - 1) / gridDim.x, uint32_t(kMinTilePaths)));
  const uint32_t tiles = uint32_t((uint64_t(numPaths) + perTile - 1) / perTile);
  if (warp == 1) next_tile(S.tiles[0], C.ticket, tiles, perTile, begin, numPaths);
  __syncthreads();
  for (int buffer = 0; S.tiles[buffer].np > 0; buffer ^= 1) {
    const PathTile &T = S.tiles[buffer];
    const int np = T.np;
    const bool apart = T.apart != 0;
    uint32_t *at = offsets + T.first;
    // the paths from a on that the stage holds together (none: a itself is too long)
    const auto batch_end = [&](int a) {
      if (T.pre[np] - T.pre[a] <= uint32_t(kStagedSegments) && !apart) return np;
      int z = a;
      while (z < np && T.pre[z + 1] - T.pre[a] <= uint32_t(kStagedSegments) && !(apart && z > a)) ++z;
      return z;
    };
    // count; the last batch's samples stay in the stage
    uint32_t total = 0, lastCount = 0;
    int lastA = 0, lastZ = 0;
    for (int a = 0; a < np;) {
      const int z = batch_end(a);
      lastA = a;
      lastZ = z;
      lastCount = z > a ? staged_samples(buffer, seg, a, z, maxDistance, fl)
                        : long_path(seg + T.begin[a], T.n(a), maxDistance, fl, nullptr, C.progress);
      total += lastCount;
      a = z > a ? z : a + 1;
    }
    if (warp == 0) {
      bool failed = false;
      const uint32_t before = samples_before(C, T.tile, total, waitLimit, &failed);
      if (threadIdx.x == 0) {
        S.base = before;
        S.failed = failed;
        if (failed) {  // this total is written after the word, the last tile's before it looks at the word
          atomicExch(C.failed, 1ull);
          __threadfence();
          offsets[numPaths] = ~0u;
        }
      }
    } else if (warp == 1) {
      next_tile(S.tiles[buffer ^ 1], C.ticket, tiles, perTile, begin, numPaths);
    }
    __syncthreads();
    if (S.failed) return;
    const uint32_t base = S.base;
    if (threadIdx.x == 0 && T.first + uint32_t(np) == numPaths) {
      at[np] = base + total;
      __threadfence();
      if (poll(C.failed) != 0) at[np] = ~0u;
    }
    const auto write_long = [&](int a, uint32_t to) {
      if (threadIdx.x == 0) at[a] = to;
      return long_path(seg + T.begin[a], T.n(a), maxDistance, fl, out + to, C.progress);
    };
    if (lastZ > lastA)
      write_staged(S, T, lastA, lastZ, base + total - lastCount, lastCount, at, out);
    else
      write_long(lastA, base + total - lastCount);
    // the batches before it once more
    uint32_t to = base;
    for (int a = 0; a < lastA;) {
      const int z = batch_end(a);
      uint32_t count;
      if (z > a) {
        count = staged_samples(buffer, seg, a, z, maxDistance, fl);
        write_staged(S, T, a, z, to, count, at, out);
      } else {
        count = write_long(a, to);
      }
      to += count;
      a = z > a ? z : a + 1;
    }
    __syncthreads();
  }
}

size_t path_counts_bytes(uint32_t numPaths) { return TileCounts::words(most_tiles(numPaths)) * sizeof(unsigned long long); }
cudaError_t launch_path_samples(const PathSegmentRecord *seg, const uint32_t *begin, uint32_t numPaths,
                                float maxDistance, PathFlags fl, PGLSampleRecord *out, uint32_t *offsets,
                                void *counts, int numSMs, cudaStream_t s, uint32_t waitLimit) {
  if (numPaths == 0) return cudaMemsetAsync(offsets, 0, sizeof(uint32_t), s);
  // once per process (thread-safe static initialisation)
  static const cudaError_t attr =
      cudaFuncSetAttribute(path_samples_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(PathShared)));
  if (attr != cudaSuccess) return attr;
  const uint32_t most = most_tiles(numPaths), blocks = uint32_t(kPathBlocksPerSM * numSMs);
  const cudaError_t e = cudaMemsetAsync(counts, 0, path_counts_bytes(numPaths), s);
  if (e != cudaSuccess) return e;
  count_launch();
  path_samples_kernel<<<most < blocks ? most : blocks, kPathThreads, sizeof(PathShared), s>>>(
      seg, begin, numPaths, maxDistance, fl, counts, waitLimit, offsets, out);
  return cudaGetLastError();
}

}  // namespace pgl
