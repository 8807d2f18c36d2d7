// Sample ingest, scene bounds, kd-tree level passes, leaf gather, the
// deterministic per-leaf ordering and the region k-nearest-neighbour table.
//
// The kd-tree is built level by level.  Samples are kept as
// (position, original index) records and, at every level, stably partitioned
// inside their node's segment (< pivot to the left, KDTreeBuilder.h:193), so
// that a node's samples stay contiguous, as in the reference's in-place
// partition (embree parallel_partition.h).  While classifying, each block
// accumulates the integer position statistics of the children it sees
// (IntegerSampleStatistics::addSample, SampleStatistics.h:261-277) in shared
// memory; because segments are contiguous a block touches few children.  The
// integer sums are order-free, so the split decisions made from them on the
// host are bit-identical to the reference's.
#include <atomic>
#include <climits>
#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include "launch.h"
#include "pgl_internal.h"

namespace pgl {

static std::atomic<unsigned long long> g_kernel_launches{0};
unsigned long long kernel_launches() { return g_kernel_launches.load(std::memory_order_relaxed); }
void count_launch() { g_kernel_launches.fetch_add(1, std::memory_order_relaxed); }



// ------------------------------------------------------------------ ingest
// Splits an AoS batch into surface / volume SoA arrays, stable within each
// class (SampleDataStorage.h:72-90).  isVol[i] is produced by pass 1.
__global__ void ingest_flag_kernel(const PGLSampleRecord *in, uint32_t n, uint32_t *isVol) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) isVol[i] = (in[i].flags & 2u) ? 1u : 0u;
}
// The same for records in host memory: each record is read once over the
// host link and kept in device memory for the scatter.
__global__ void ingest_flag_stage_kernel(const PGLSampleRecord *in, uint32_t n, uint32_t *isVol,
                                         PGLSampleRecord *stage) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const PGLSampleRecord r = in[i];
  stage[i] = r;
  isVol[i] = (r.flags & 2u) ? 1u : 0u;
}
__global__ void ingest_scatter_kernel(const PGLSampleRecord *in, uint32_t n, const uint32_t *volRank,
                                      float4 *sP, float4 *sD, float *sPdf, uint32_t *sFlags, uint64_t sBase,
                                      float4 *vP, float4 *vD, float *vPdf, uint32_t *vFlags, uint64_t vBase) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  PGLSampleRecord r = in[i];
  uint32_t vr = volRank[i];
  float4 p = make_float4(r.px, r.py, r.pz, r.distance);
  float4 d = make_float4(r.dx, r.dy, r.dz, r.weight);
  if (r.flags & 2u) {
    uint64_t o = vBase + vr;
    vP[o] = p; vD[o] = d; vPdf[o] = r.pdf; vFlags[o] = r.flags;
  } else {
    uint64_t o = sBase + (i - vr);
    sP[o] = p; sD[o] = d; sPdf[o] = r.pdf; sFlags[o] = r.flags;
  }
}
__global__ void export_kernel(const float4 *P, const float4 *D, const float *pdf, const uint32_t *flags, uint64_t n,
                              PGLSampleRecord *out) {
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = P[i], d = D[i];
  PGLSampleRecord r{p.x, p.y, p.z, d.x, d.y, d.z, d.w, pdf[i], p.w, flags[i]};
  out[i] = r;
}

// ------------------------------------------------------------------ bounds
// min/max of positions [0, n) (the caller passes n-1: Field.h:326-344 stops
// one short of the end).  Floats are mapped to order-preserving integers.
__device__ __forceinline__ uint32_t ford(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unford(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? o & 0x7FFFFFFFu : ~o);
}
// Bounds of the positions as ordered integers.  Bytes bound (1.5M positions in
// 7 us) with six atomics per block; with six per warp they took 130 us.
__global__ void __launch_bounds__(256) bounds_kernel(const float4 *P, uint64_t n, uint32_t *out6) {
  __shared__ uint32_t part[8][6];
  uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0, 0, 0};
#pragma unroll 4
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    float4 p = P[i];
    float c[3] = {p.x, p.y, p.z};
    for (int d = 0; d < 3; ++d) {
      uint32_t o = ford(c[d]);
      lo[d] = min(lo[d], o);
      hi[d] = max(hi[d], o);
    }
  }
  for (int d = 0; d < 3; ++d) {
    lo[d] = __reduce_min_sync(0xFFFFFFFFu, lo[d]);
    hi[d] = __reduce_max_sync(0xFFFFFFFFu, hi[d]);
  }
  if ((threadIdx.x & 31) == 0)
    for (int d = 0; d < 3; ++d) {
      part[threadIdx.x >> 5][d] = lo[d];
      part[threadIdx.x >> 5][3 + d] = hi[d];
    }
  __syncthreads();
  if (threadIdx.x < 6) {
    uint32_t v = part[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) {
      const uint32_t o = part[w][threadIdx.x];
      v = threadIdx.x < 3 ? min(v, o) : max(v, o);
    }
    if (threadIdx.x < 3) atomicMin(&out6[threadIdx.x], v);
    else atomicMax(&out6[threadIdx.x], v);
  }
}

// ------------------------------------------------------------------ kd levels
// One job per inner node visited at the current level.

constexpr int kKdThreads = 256;
constexpr int kKdItems = 8;                       // samples per thread
constexpr int kKdTile = kKdThreads * kKdItems;    // samples per block

// A sample's place in its node's frame in units of 1 / 4096, before and after
// the conversion to integers (in 32 bits where that holds them: the 64-bit
// conversion runs at a fraction of the rate: with it the root's statistics took
// 22 us of 1.5M samples in place of 12, 62 us with an atomic per warp).
__device__ __noinline__ long long to_int64(float t) { return (long long)t; }
__device__ __forceinline__ void quantize(const KdJob &j, float4 p, float t[3], long long q[3], long long qv[3]) {
  float c[3] = {p.x, p.y, p.z}, tv[3];
  bool small = true;
  for (int d = 0; d < 3; ++d) {
    t[d] = (c[d] - j.c[d]) * j.inv[d];
    tv[d] = (t[d] * t[d]) * 4096.f;
    t[d] *= 4096.f;
    small = small && fabsf(t[d]) < 0x1p31f && tv[d] < 0x1p31f;
  }
  if (small) {
    for (int d = 0; d < 3; ++d) {
      q[d] = __float2int_rz(t[d]);
      qv[d] = __float2int_rz(tv[d]);
    }
  } else {
    for (int d = 0; d < 3; ++d) {
      q[d] = to_int64(t[d]);
      qv[d] = to_int64(tv[d]);
    }
  }
}

// Adds one sample's integer statistics (or a warp's reduced ones) to an
// accumulator in shared or global memory.
__device__ __forceinline__ void acc_add(IStatsAcc *a, const long long m[3], const long long v[3], const long long lo[3],
                                        const long long hi[3], unsigned long long n) {
  for (int d = 0; d < 3; ++d) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&a->m[d]), (unsigned long long)m[d]);
    atomicAdd(reinterpret_cast<unsigned long long *>(&a->v[d]), (unsigned long long)v[d]);
    atomicMin(&a->lo[d], lo[d]);
    atomicMax(&a->hi[d], hi[d]);
  }
  atomicAdd(&a->n, n);
}

// Smallest and largest integers of some samples by their unconverted floats (the
// conversion keeps the order; a NaN converts to the smallest integer, infinities
// to the ends, which are also what no samples leave).
struct FloatRange {
  float lo, hi;
  __device__ __forceinline__ void clear() {
    lo = INFINITY;
    hi = -INFINITY;
  }
  __device__ __forceinline__ void add(float t, bool on) {
    lo = fminf(lo, on ? (t == t ? t : -INFINITY) : INFINITY);
    hi = fmaxf(hi, on ? t : -INFINITY);
  }
  __device__ __forceinline__ void warp(long long &l, long long &h) const {
    l = (long long)unford(__reduce_min_sync(0xFFFFFFFFu, ford(lo)));
    h = (long long)unford(__reduce_max_sync(0xFFFFFFFFu, ford(hi)));
  }
};
// A warp's running integer statistics of one job: sums over all samples and
// over the left ones per lane, ranges of both sides per lane, counts per warp.
struct WarpSideAcc {
  long long m[3], v[3], ml[3], vl[3];
  FloatRange range[2][3];
  uint32_t n, nl;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      m[d] = v[d] = ml[d] = vl[d] = 0;
      range[0][d].clear();
      range[1][d].clear();
    }
    n = nl = 0;
  }
};
__device__ __forceinline__ long long warp_sum64(long long x) {
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, off);
  return x;
}
// A warp's reduced statistics of a job: both sides' IStatsAcc as 26 words.
constexpr int kAccWords = sizeof(IStatsAcc) / 8;
static_assert(kAccWords == 13 && offsetof(IStatsAcc, v) == 24 && offsetof(IStatsAcc, lo) == 48 &&
                  offsetof(IStatsAcc, hi) == 72 && offsetof(IStatsAcc, n) == 96,
              "words of m, v, lo, hi, n");
struct WarpWords {
  IStatsAcc side[2];
  uint32_t job;  // ~0: none
  bool stats;
};
// Reduces a warp's running statistics into `out` and clears them.
__device__ __forceinline__ void warp_words(WarpSideAcc &w, uint32_t job, bool stats, WarpWords &out) {
  const int lane = threadIdx.x & 31;
  if (stats) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const long long m = warp_sum64(w.m[d]), ml = warp_sum64(w.ml[d]);
      const long long v = warp_sum64(w.v[d]), vl = warp_sum64(w.vl[d]);
      long long lo[2], hi[2];
      w.range[0][d].warp(lo[0], hi[0]);
      w.range[1][d].warp(lo[1], hi[1]);
      if (lane == 0) {
        out.side[0].m[d] = ml;
        out.side[0].v[d] = vl;
        out.side[1].m[d] = m - ml;
        out.side[1].v[d] = v - vl;
        for (int sd = 0; sd < 2; ++sd) {
          out.side[sd].lo[d] = lo[sd];
          out.side[sd].hi[d] = hi[sd];
        }
      }
    }
  }
  if (lane == 0) {
    out.side[0].n = w.nl;
    out.side[1].n = w.n - w.nl;
    out.job = job;
    out.stats = stats;
  }
  w.clear();
  __syncwarp();
}
// Word k of the job's two accumulators takes the warps' words: atomics in
// global memory, which are single operations there (64-bit ones in shared memory
// are loops).  The warps [w, end) of `words` that hold w's job.
__device__ __forceinline__ void add_words(const WarpWords *words, int w, int end, int k, IStatsAcc *acc) {
  const uint32_t job = words[w].job;
  const int side = k / kAccWords, f = k % kAccWords;
  if (!words[w].stats && f != kAccWords - 1) return;
  unsigned long long n = 0;
  long long x = 0;
  for (int o = w; o < end; ++o) {
    const WarpWords &W = words[o];
    if (W.job != job || W.side[side].n == 0) continue;
    const long long y = reinterpret_cast<const long long *>(&W.side[side])[f];
    if (n == 0) x = y;
    else if (f >= 9 && f < 12) x = max(x, y);
    else if (f >= 6 && f < 9) x = min(x, y);
    else x += y;
    n += W.side[side].n;
  }
  if (n == 0) return;
  long long *to = reinterpret_cast<long long *>(&acc[2 * job + uint32_t(side)]) + f;
  if (f >= 9 && f < 12) atomicMax(to, x);
  else if (f >= 6 && f < 9) atomicMin(to, x);
  else atomicAdd(reinterpret_cast<unsigned long long *>(to), (unsigned long long)x);
}

// Classifies the samples of every job at this level: side flag (1 = left),
// child statistics into acc[2*job + side].  jobOf[i] is the job of sample i
// (or ~0 when the sample already sits in a finished leaf).  Samples of a job
// are contiguous, so a warp mostly meets one job: each lane keeps running
// statistics of the warp's current job in registers, and the warp reduces
// and adds them only when its job changes and, together with the other warps of
// the block, at the end.  Samples past the fourth job of 32 add one by one.
// Latency bound.  1.5M samples: 48 us with 64-bit shared-memory atomics (loops)
// per warp, 64-bit conversions and the ranges in integers, 27 us so.
__global__ void __launch_bounds__(kKdThreads, 3)
kd_classify_kernel(const float4 *pos, const uint32_t *jobOf, uint32_t n, const KdJob *jobs, uint32_t *isLeft,
                   IStatsAcc *acc) {
  __shared__ WarpWords words[kKdThreads / 32];
  const uint32_t tileBegin = blockIdx.x * kKdTile;
  if (tileBegin >= n) return;
  const uint32_t tileEnd = min(n, tileBegin + kKdTile);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned full = 0xFFFFFFFFu;
  WarpSideAcc w;
  w.clear();
  uint32_t cur = ~0u;  // the warp's current job
  bool curStats = false;
  KdJob j;
  uint32_t jAt = ~0u;  // the job in j
  // two samples ahead
  uint32_t i = tileBegin + threadIdx.x, jidA = ~0u, jidB = ~0u;
  float4 pA = make_float4(0.0f, 0.0f, 0.0f, 0.0f), pB = pA;
  if (i < tileEnd) {
    jidA = jobOf[i];
    pA = pos[i];
  }
  if (i + kKdThreads < tileEnd) {
    jidB = jobOf[i + kKdThreads];
    pB = pos[i + kKdThreads];
  }
#pragma unroll 1
  for (uint32_t base = tileBegin; base < tileEnd; base += kKdThreads, i += kKdThreads) {
    const uint32_t jid = jidA;
    const float4 p = pA;
    jidA = jidB;
    pA = pB;
    jidB = ~0u;
    if (i + 2 * kKdThreads < tileEnd) {
      jidB = jobOf[i + 2 * kKdThreads];
      pB = pos[i + 2 * kKdThreads];
    }
    uint32_t left = 0;
    float t[3] = {0.0f, 0.0f, 0.0f};
    long long q[3] = {0, 0, 0}, qv[3] = {0, 0, 0};
    bool stats = false;
    if (jid != ~0u) {
      if (jid != jAt) {
        j = jobs[jid];
        jAt = jid;
      }
      const float coord = j.dim == 0 ? p.x : (j.dim == 1 ? p.y : p.z);
      left = coord < j.pos ? 1u : 0u;
      stats = j.needStats != 0;
      if (stats) quantize(j, p, t, q, qv);
    }
    if (i < tileEnd) isLeft[i] = left;
    unsigned rest = __ballot_sync(full, jid != ~0u);
#pragma unroll 1
    for (int g = 0; g < 4 && rest != 0; ++g) {
      const int src = __ffs(rest) - 1;
      const uint32_t j0 = __shfl_sync(full, jid, src);
      if (j0 != cur) {
        if (cur != ~0u) {
          warp_words(w, cur, curStats, words[warp]);
          if (lane < 2 * kAccWords) add_words(words, warp, warp + 1, lane, acc);
          __syncwarp();
        }
        cur = j0;
        curStats = __shfl_sync(full, stats ? 1 : 0, src) != 0;
      }
      const bool on = jid == j0, onLeft = on && left != 0u;
      const unsigned members = __ballot_sync(full, on);
      w.n += __popc(members);
      w.nl += __popc(__ballot_sync(full, onLeft));
      rest &= ~members;
      if (curStats) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          w.m[d] += on ? q[d] : 0ll;
          w.v[d] += on ? qv[d] : 0ll;
          w.ml[d] += onLeft ? q[d] : 0ll;
          w.vl[d] += onLeft ? qv[d] : 0ll;
          w.range[0][d].add(t[d], onLeft);
          w.range[1][d].add(t[d], on && !onLeft);
        }
      }
    }
    if (rest >> lane & 1u) {
      IStatsAcc *a = &acc[2 * jid + (left ? 0u : 1u)];
      if (stats) acc_add(a, q, qv, q, q, 1ull);
      else atomicAdd(&a->n, 1ull);
    }
  }
  warp_words(w, cur, curStats, words[warp]);
  __syncthreads();
  // the first warp of each job adds for all that hold it
  if (cur != ~0u) {
    for (int o = 0; o < warp; ++o)
      if (words[o].job == cur) return;
    if (lane < 2 * kAccWords) add_words(words, warp, kKdThreads / 32, lane, acc);
  }
}

// Integer statistics of all samples relative to the root bounds (the root is
// a leaf: KDTreeBuilder.h:94-115).
__global__ void __launch_bounds__(kKdThreads)
kd_root_stats_kernel(const float4 *pos, uint32_t n, KdJob job, IStatsAcc *acc) {
  __shared__ WarpWords words[kKdThreads / 32];
  long long m[3] = {0, 0, 0}, v[3] = {0, 0, 0}, lo[3], hi[3];
  FloatRange range[3];
  for (int d = 0; d < 3; ++d) range[d].clear();
  uint32_t cnt = 0;
#pragma unroll 4
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float t[3];
    long long q[3], qv[3];
    quantize(job, pos[i], t, q, qv);
    for (int d = 0; d < 3; ++d) {
      m[d] += q[d];
      v[d] += qv[d];
      range[d].add(t[d], true);
    }
    cnt++;
  }
  for (int d = 0; d < 3; ++d) {
    m[d] = warp_sum64(m[d]);
    v[d] = warp_sum64(v[d]);
    range[d].warp(lo[d], hi[d]);
  }
  cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
  if ((threadIdx.x & 31) == 0) {
    WarpWords &W = words[threadIdx.x >> 5];
    for (int d = 0; d < 3; ++d) {
      W.side[0].m[d] = m[d];
      W.side[0].v[d] = v[d];
      W.side[0].lo[d] = lo[d];
      W.side[0].hi[d] = hi[d];
    }
    W.side[0].n = cnt;
    W.job = 0;
    W.stats = true;
  }
  __syncthreads();
  if (threadIdx.x < kAccWords) add_words(words, 0, kKdThreads / 32, threadIdx.x, acc);
}

// One pass down an existing tree: the leaf every sample reaches, by the
// builder's rule (coord < split goes left, KDTreeBuilder.h:193), as the
// leaf's slot (key) beside the sample's index (val).
__global__ void kd_route_kernel(const float4 *pos, uint32_t n, const KDNode *nodes, const uint32_t *nodeSlot,
                                uint32_t *key, uint32_t *val) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 p = pos[i];
  uint32_t nd = 0;
  KDNode node = nodes[0];
  while ((node.bits >> 30) != 3u) {
    const uint32_t dim = node.bits >> 30;
    const float c = dim == 0 ? p.x : (dim == 1 ? p.y : p.z);
    nd = (node.bits & 0x3FFFFFFFu) + (c < node.split ? 0u : 1u);
    node = nodes[nd];
  }
  key[i] = nodeSlot[nd];
  val[i] = i;
}
// Samples in slot order: positions and their leaf nodes.
__global__ void kd_route_gather_kernel(const float4 *pos, const uint32_t *key, const uint32_t *val, uint32_t n,
                                       const uint32_t *slotNode, float4 *posOut, uint32_t *nodeOut) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  posOut[j] = pos[val[j]];
  nodeOut[j] = slotNode[key[j]];
}

// Stable partition inside each job's segment using the exclusive scan of the
// left flags; finished samples keep their place.
__global__ void kd_scatter_kernel(const float4 *pos, const uint32_t *jobOf, const uint32_t *isLeft,
                                  const uint32_t *scanLeft, uint32_t n, const KdJob *jobs, float4 *posOut,
                                  uint32_t *nodeOut) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t jid = jobOf[i];
  if (jid == ~0u) {
    posOut[i] = pos[i];
    nodeOut[i] = ~0u;
    return;
  }
  const KdJob j = jobs[jid];
  uint32_t leftBefore = scanLeft[i] - scanLeft[j.begin];
  uint32_t L = scanLeft[j.end - 1] + isLeft[j.end - 1] - scanLeft[j.begin];
  uint32_t dst;
  uint32_t child;
  if (isLeft[i]) {
    dst = j.begin + leftBefore;
    child = j.left;
  } else {
    dst = j.begin + L + (i - j.begin - leftBefore);
    child = j.left + 1;
  }
  posOut[dst] = pos[i];
  nodeOut[dst] = child;
}

// Maps each sample's node to the job index of the next level (~0 if the node
// is a finished leaf).
// The job of every sample of a level (~0 for samples in finished leaves), and
// the level's child accumulators cleared, in one launch.
__global__ void kd_job_of_kernel(const uint32_t *node, uint32_t n, const uint32_t *nodeToJob, uint32_t *jobOf,
                                 IStatsAcc *acc, uint32_t accCount) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < accCount) {
    IStatsAcc a;
    for (int d = 0; d < 3; ++d) { a.m[d] = 0; a.v[d] = 0; a.lo[d] = LLONG_MAX; a.hi[d] = LLONG_MIN; }
    a.n = 0;
    acc[i] = a;
  }
  if (i >= n) return;
  uint32_t nd = node[i];
  jobOf[i] = nd == ~0u ? ~0u : nodeToJob[nd];
}

// ------------------------------------------------------------------ gather + ordering
// Gathers full samples into leaf order.
__global__ void gather_kernel(const float4 *posIdx, uint32_t n, const float4 *P, const float4 *D, const float *pdf,
                              float4 *oP, float4 *oD, float *oPdf) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t src = __float_as_uint(posIdx[i].w);
  oP[i] = P[src];
  oD[i] = D[src];
  oPdf[i] = pdf[src];
}
// 64-bit sort keys of the samples in leaf order, beside the samples' indices:
// the leaf's ordinal, then the weight's bits mapped to an order-preserving
// integer (-0 as +0), the first field of SampleDataLess (SampleData.h:82-93).
// blockIdx.x: leaf, blockIdx.y: its part.  Bound by the scattered reads: 1.5M
// samples 15 us, the permutation below 34 us; with the full samples gathered
// first and a block per leaf the three kernels took 35 + 31 + 29 us (56 for the
// second with large leaves).
__global__ void leaf_key_kernel(const float4 *posIdx, const uint32_t *leafBegin, const uint32_t *leafEnd,
                                const float4 *D, unsigned long long *key64, uint32_t *val) {
  const uint32_t leaf = blockIdx.x, end = leafEnd[leaf];
  const unsigned long long hi = (unsigned long long)leaf << 32;
  for (uint32_t i = leafBegin[leaf] + blockIdx.y * blockDim.x + threadIdx.x; i < end; i += gridDim.y * blockDim.x) {
    const uint32_t src = __float_as_uint(posIdx[i].w);
    const float w = D[src].w;
    key64[i] = hi | ford(w == 0.0f ? 0.0f : w);
    val[i] = src;
  }
}
__device__ __forceinline__ bool sample_less(float4 pa, float4 da, float fa, float4 pb, float4 db, float fb) {
  if (da.w != db.w) return da.w < db.w;   // weight
  if (fa != fb) return fa < fb;           // pdf
  if (pa.w != pb.w) return pa.w < pb.w;   // distance
  if (pa.x != pb.x) return pa.x < pb.x;
  if (pa.y != pb.y) return pa.y < pb.y;
  if (pa.z != pb.z) return pa.z < pb.z;
  if (da.x != db.x) return da.x < db.x;
  if (da.y != db.y) return da.y < db.y;
  return da.z < db.z;
}
// Permutes the samples into the sorted order (all samples, one thread each).
__global__ void permute_kernel(const uint32_t *sortedVal, uint32_t n, const float4 *P, const float4 *D,
                               const float *pdf, float4 *oP, float4 *oD, float *oPdf) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = sortedVal[i];
  oP[i] = P[s];
  oD[i] = D[s];
  oPdf[i] = pdf[s];
}
// Ties of equal weight within a leaf (equal adjacent 64-bit keys: same leaf,
// same weight) are ordered by the full comparator.  Float weights collide by
// chance (a few percent of the samples of a 2M batch), in runs of a handful,
// so every run is sorted by the thread at its first sample, all runs at once.
__global__ void fix_ties_kernel(const unsigned long long *sortedKey, uint32_t n, float4 *oP, float4 *oD,
                                float *oPdf) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i + 1 >= n) return;
  const unsigned long long k = sortedKey[i];
  if (sortedKey[i + 1] != k || (i > 0 && sortedKey[i - 1] == k)) return;  // not the start of a run
  uint32_t j = i + 2;
  while (j < n && sortedKey[j] == k) ++j;
  for (uint32_t x = i + 1; x < j; ++x) {  // insertion sort of the run [i, j)
    float4 kp = oP[x], kd = oD[x];
    float kf = oPdf[x];
    uint32_t y = x;
    while (y > i && sample_less(kp, kd, kf, oP[y - 1], oD[y - 1], oPdf[y - 1])) {
      oP[y] = oP[y - 1];
      oD[y] = oD[y - 1];
      oPdf[y] = oPdf[y - 1];
      --y;
    }
    oP[y] = kp;
    oD[y] = kd;
    oPdf[y] = kf;
  }
}

// ------------------------------------------------------------------ regions
__global__ void copy_region_kernel(RegionDir *regions, const uint32_t *dst, const uint32_t *src, uint32_t n) {
  uint32_t k = blockIdx.x;
  if (k >= n) return;
  const uint32_t *s = reinterpret_cast<const uint32_t *>(&regions[src[k]]);
  uint32_t *d = reinterpret_cast<uint32_t *>(&regions[dst[k]]);
  for (uint32_t i = threadIdx.x; i < sizeof(RegionDir) / 4; i += blockDim.x) d[i] = s[i];
}

// 8 nearest region means per region (KNN.h:212-266); nanoflann's squared
// distance ((dx*dx + dy*dy) + dz*dz), ties by region index.
__device__ __forceinline__ float mean_distance(float4 q, float4 p) {
  float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
  float d = 0.0f;
  d += dx * dx;
  d += dy * dy;
  d += dz * dz;
  return d;
}
// by one thread, any distances
__device__ __noinline__ int nearest_in_order(const float4 *means, uint32_t R, float4 q, uint32_t bi[8]) {
  float bd[8];
  int cnt = 0;
  for (uint32_t j = 0; j < R; ++j) {
    const float d = mean_distance(q, means[j]);
    if (cnt < 8 || d < bd[cnt - 1]) {
      int k = cnt < 8 ? cnt : 7;
      while (k > 0 && bd[k - 1] > d) {
        if (k < 8) { bd[k] = bd[k - 1]; bi[k] = bi[k - 1]; }
        --k;
      }
      bd[k] = d;
      bi[k] = j;
      if (cnt < 8) cnt++;
    }
  }
  return cnt;
}
// A warp per region: each lane keeps the nearest 8 of every 32nd mean, then the
// warp takes the least of the lanes' heads 8 times.  With distances that have no
// order (infinite or NaN means) lane 0 goes through the means alone.  128
// regions: 68 us with a thread per region, 5 us so.
__global__ void __launch_bounds__(128) knn_kernel(const float4 *means, uint32_t R, Neighbours *out) {
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xFFFFFFFFu;
  if (r >= R) return;
  const float4 q = means[r];
  float bd[8];
  uint32_t bi[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    bd[k] = INFINITY;
    bi[k] = ~0u;
  }
  bool odd = false;
  for (uint32_t j = lane; j < R; j += 32) {
    const float d = mean_distance(q, means[j]);
    odd = odd || !(d <= FLT_MAX);
    if (!(d < bd[7])) continue;
#pragma unroll
    for (int k = 7; k > 0; --k) {
      const bool down = d < bd[k - 1], here = d < bd[k];
      bi[k] = down ? bi[k - 1] : (here ? j : bi[k]);
      bd[k] = down ? bd[k - 1] : (here ? d : bd[k]);
    }
    if (d < bd[0]) {
      bd[0] = d;
      bi[0] = j;
    }
  }
  uint32_t mine = ~0u;  // lane k < 8: neighbour k
  int cnt = int(min(R, 8u));
  if (__any_sync(full, odd)) {
    uint32_t in[8];
    for (int k = 0; k < 8; ++k) in[k] = ~0u;
    if (lane == 0) cnt = nearest_in_order(means, R, q, in);
    cnt = __shfl_sync(full, cnt, 0);
    for (int k = 0; k < 8; ++k) {
      const uint32_t id = __shfl_sync(full, in[k], 0);
      if (lane == k) mine = id;
    }
  } else {
    for (int k = 0; k < 8; ++k) {
      const uint32_t d = __reduce_min_sync(full, __float_as_uint(bd[0]));  // not negative
      const uint32_t id = __reduce_min_sync(full, __float_as_uint(bd[0]) == d ? bi[0] : ~0u);
      if (lane == k) mine = id;
      if (bi[0] == id && id != ~0u) {
#pragma unroll
        for (int m = 0; m < 7; ++m) {
          bd[m] = bd[m + 1];
          bi[m] = bi[m + 1];
        }
        bd[7] = INFINITY;
        bi[7] = ~0u;
      }
    }
  }
  if (lane == 0) out[r].size = uint32_t(cnt);
  if (lane < 8) {
    const float4 p = lane < cnt ? means[mine] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    out[r].ids[lane] = lane < cnt ? mine : ~0u;
    out[r].px[lane] = p.x;
    out[r].py[lane] = p.y;
    out[r].pz[lane] = p.z;
  }
}

// ------------------------------------------------------------------ launchers
PGL_DEFINE_TABLE_UPLOAD(spatial_upload_tables)

cudaError_t scratch_reserve(Scratch &s, size_t bytes) {
  if (bytes <= s.bytes && s.ptr) return cudaSuccess;
  if (s.ptr) cudaFree(s.ptr);
  s.ptr = nullptr;
  s.bytes = 0;
  size_t want = bytes < 256 ? 256 : bytes + bytes / 4;
  cudaError_t e = cudaMalloc(&s.ptr, want);
  if (e == cudaSuccess) s.bytes = want;
  return e;
}
void scratch_free(Scratch &s) {
  if (s.ptr) cudaFree(s.ptr);
  s.ptr = nullptr;
  s.bytes = 0;
}

static inline unsigned blocks_for(uint64_t n, unsigned t) { return unsigned((n + t - 1) / t); }

cudaError_t ingest_samples(const PGLSampleRecord *in, uint32_t n, Scratch &scratch, SoAView surf, SoAView vol,
                           uint32_t *numVolume, cudaStream_t s, PGLSampleRecord *stage) {
  if (n == 0) { *numVolume = 0; return cudaSuccess; }
  size_t tempBytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tempBytes, (uint32_t *)nullptr, (uint32_t *)nullptr, int(n), s);
  const size_t flagBytes = (size_t(n) + 1) * sizeof(uint32_t);
  const size_t off = (flagBytes * 2 + 255) / 256 * 256;
  cudaError_t e = scratch_reserve(scratch, off + tempBytes);
  if (e != cudaSuccess) return e;
  uint32_t *isVol = reinterpret_cast<uint32_t *>(scratch.ptr);
  uint32_t *rank = isVol + (n + 1);
  void *temp = static_cast<char *>(scratch.ptr) + off;
  count_launch();
  if (stage) {
    ingest_flag_stage_kernel<<<blocks_for(n, 256), 256, 0, s>>>(in, n, isVol, stage);
    in = stage;
  } else {
    ingest_flag_kernel<<<blocks_for(n, 256), 256, 0, s>>>(in, n, isVol);
  }
  cub::DeviceScan::ExclusiveSum(temp, tempBytes, isVol, rank, int(n), s);
  count_launch();
  ingest_scatter_kernel<<<blocks_for(n, 256), 256, 0, s>>>(in, n, rank, surf.P, surf.D, surf.pdf, surf.flags, surf.base,
                                                          vol.P, vol.D, vol.pdf, vol.flags, vol.base);
  uint32_t last[2];
  cudaMemcpyAsync(&last[0], rank + n - 1, 4, cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(&last[1], isVol + n - 1, 4, cudaMemcpyDeviceToHost, s);
  e = cudaStreamSynchronize(s);
  *numVolume = last[0] + last[1];
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t export_samples(const float4 *P, const float4 *D, const float *pdf, const uint32_t *flags, uint64_t n,
                           PGLSampleRecord *out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  export_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P, D, pdf, flags, n, out);
  return cudaGetLastError();
}

cudaError_t scene_bounds(const float4 *P, uint64_t n, uint32_t *d6, cudaStream_t s) {
  uint32_t init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
  cudaError_t e = cudaMemcpyAsync(d6, init, sizeof(init), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess || n == 0) return e;
  unsigned b = blocks_for(n, 1024);
  if (b > 1024) b = 1024;
  count_launch();
  bounds_kernel<<<b, 256, 0, s>>>(P, n, d6);
  return cudaGetLastError();
}

__global__ void init_posidx_kernel(const float4 *P, uint32_t n, float4 *posIdx) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = P[i];
  posIdx[i] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
}
cudaError_t init_posidx(const float4 *P, uint32_t n, float4 *posIdx, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  init_posidx_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P, n, posIdx);
  return cudaGetLastError();
}

__global__ void init_acc_kernel(IStatsAcc *acc, uint32_t count) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  IStatsAcc a;
  for (int d = 0; d < 3; ++d) { a.m[d] = 0; a.v[d] = 0; a.lo[d] = LLONG_MAX; a.hi[d] = LLONG_MIN; }
  a.n = 0;
  acc[i] = a;
}
cudaError_t init_acc(IStatsAcc *acc, uint32_t count, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  count_launch();
  init_acc_kernel<<<blocks_for(count, 128), 128, 0, s>>>(acc, count);
  return cudaGetLastError();
}

cudaError_t kd_root_stats(const float4 *pos, uint32_t n, const KdJob &job, IStatsAcc *acc, cudaStream_t s) {
  unsigned b = blocks_for(n, kKdThreads * 8);
  if (b < 1) b = 1;
  if (b > 608) b = 608;
  count_launch();
  kd_root_stats_kernel<<<b, kKdThreads, 0, s>>>(pos, n, job, acc);
  return cudaGetLastError();
}

cudaError_t kd_job_of(const uint32_t *node, uint32_t n, const uint32_t *nodeToJob, uint32_t *jobOf, IStatsAcc *acc,
                      uint32_t accCount, cudaStream_t s) {
  const uint32_t m = n > accCount ? n : accCount;
  if (m == 0) return cudaSuccess;
  count_launch();
  kd_job_of_kernel<<<blocks_for(m, 256), 256, 0, s>>>(node, n, nodeToJob, jobOf, acc, accCount);
  return cudaGetLastError();
}

cudaError_t kd_level(const float4 *pos, const uint32_t *jobOf, uint32_t n, const KdJob *jobs, uint32_t *isLeft,
                     uint32_t *scanLeft, IStatsAcc *acc, float4 *posOut, uint32_t *nodeOut, Scratch &scratch,
                     cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  kd_classify_kernel<<<blocks_for(n, kKdTile), kKdThreads, 0, s>>>(pos, jobOf, n, jobs, isLeft, acc);
  size_t tempBytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tempBytes, isLeft, scanLeft, int(n), s);
  cudaError_t e = scratch_reserve(scratch, tempBytes);
  if (e != cudaSuccess) return e;
  cub::DeviceScan::ExclusiveSum(scratch.ptr, tempBytes, isLeft, scanLeft, int(n), s);
  count_launch();
  kd_scatter_kernel<<<blocks_for(n, 256), 256, 0, s>>>(pos, jobOf, isLeft, scanLeft, n, jobs, posOut, nodeOut);
  return cudaGetLastError();
}

cudaError_t kd_route(const float4 *pos, uint32_t n, const KDNode *nodes, const uint32_t *nodeSlot, uint32_t numSlots,
                     const uint32_t *slotNode, uint32_t *keys, uint32_t *vals, uint32_t *keysB, uint32_t *valsB,
                     float4 *posOut, uint32_t *nodeOut, Scratch &scratch, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  kd_route_kernel<<<blocks_for(n, 256), 256, 0, s>>>(pos, n, nodes, nodeSlot, keys, vals);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  int bits = 1;
  while (bits < 32 && (1u << bits) < numSlots) ++bits;
  cub::DoubleBuffer<uint32_t> k(keys, keysB), v(vals, valsB);
  size_t tempBytes = 0;
  e = cub::DeviceRadixSort::SortPairs(nullptr, tempBytes, k, v, int(n), 0, bits, s);
  if (e != cudaSuccess) return e;
  e = scratch_reserve(scratch, tempBytes);
  if (e != cudaSuccess) return e;
  e = cub::DeviceRadixSort::SortPairs(scratch.ptr, tempBytes, k, v, int(n), 0, bits, s);
  if (e != cudaSuccess) return e;
  count_launch();
  kd_route_gather_kernel<<<blocks_for(n, 256), 256, 0, s>>>(pos, k.Current(), v.Current(), n, slotNode, posOut,
                                                              nodeOut);
  return cudaGetLastError();
}
cudaError_t kd_classify(const float4 *pos, const uint32_t *jobOf, uint32_t n, const KdJob *jobs, uint32_t *isLeft,
                        IStatsAcc *acc, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  kd_classify_kernel<<<blocks_for(n, kKdTile), kKdThreads, 0, s>>>(pos, jobOf, n, jobs, isLeft, acc);
  return cudaGetLastError();
}

cudaError_t gather_and_order(const float4 *posIdx, uint32_t n, const float4 *P, const float4 *D, const float *pdf,
                             const uint32_t *leafBegin, uint32_t numLeaves, bool sorted,
                             uint32_t *vals, unsigned long long *keys64, float4 *oP, float4 *oD, float *oPdf, Scratch &scratch,
                             cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (!sorted) {
    count_launch();
    gather_kernel<<<blocks_for(n, 256), 256, 0, s>>>(posIdx, n, P, D, pdf, oP, oD, oPdf);
    return cudaGetLastError();
  }
  // stable order by (leaf, weight key): one LSD radix sort over the bits in
  // use (the leaves' sample ranges are disjoint and cover [0, n))
  uint32_t *valsOut = vals + n;
  unsigned long long *keys64Out = keys64 + n;
  const uint32_t *ends = leafBegin + numLeaves;  // caller stores ends after begins
  // blocks for about eight samples per thread whatever the number of leaves
  uint32_t parts = n / 2048 / numLeaves;
  parts = parts < 1 ? 1 : (parts > 4096 ? 4096 : parts);
  count_launch();
  leaf_key_kernel<<<dim3(numLeaves, parts), 256, 0, s>>>(posIdx, leafBegin, ends, D, keys64, vals);
  int leafBits = 1;
  while (leafBits < 32 && (1u << leafBits) < numLeaves) ++leafBits;
  size_t tempBytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tempBytes, keys64, keys64Out, vals, valsOut, int(n), 0, 32 + leafBits, s);
  cudaError_t e = scratch_reserve(scratch, tempBytes);
  if (e != cudaSuccess) return e;
  cub::DeviceRadixSort::SortPairs(scratch.ptr, tempBytes, keys64, keys64Out, vals, valsOut, int(n), 0, 32 + leafBits,
                                  s);
  count_launch();
  permute_kernel<<<blocks_for(n, 256), 256, 0, s>>>(valsOut, n, P, D, pdf, oP, oD, oPdf);
  count_launch();
  fix_ties_kernel<<<blocks_for(n, 256), 256, 0, s>>>(keys64Out, n, oP, oD, oPdf);
  return cudaGetLastError();
}

cudaError_t copy_regions(RegionDir *regions, const uint32_t *dst, const uint32_t *src, uint32_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  copy_region_kernel<<<n, 256, 0, s>>>(regions, dst, src, n);
  return cudaGetLastError();
}

cudaError_t build_knn(const float4 *means, uint32_t R, Neighbours *out, cudaStream_t s) {
  if (R == 0) return cudaSuccess;
  count_launch();
  knn_kernel<<<blocks_for(uint64_t(R) * 32, 128), 128, 0, s>>>(means, R, out);
  return cudaGetLastError();
}

}  // namespace pgl
