// Directional quadtree field type: the per-region fit and update of
// DirectionalQuadtreeFactory (directional/dqt/DQTFactory.h:149-324) on the
// device, one thread block per region, regions handed out by an atomic queue.
//
// An update (DQTFactory.h:199-281) splats every sample of the region, in the
// region's sample order, into the leaves of the current statistics tree: a
// box of footprintFactor times the size of the leaf the sample's point falls
// in, clipped to the unit square, gives each leaf it overlaps the overlap's
// share of the box.  Per chunk of samples each thread maps one sample to the
// square (the passes of a fit after the first read the points back), finds its
// box and the leaves it overlaps; then threads own leaves and add the shares in
// sample order, so every leaf's sums are the reference's sequential sums:
//   few leaves (the first passes of a fit): the samples write a leaf x sample
//   matrix of shares, and three threads per leaf each run down its row;
//   more: masks of the samples that overlap each leaf give every pair of a
//   leaf and a sample a slot in leaf and sample order, the samples write share,
//   share x first and share x second moment there and a thread per leaf adds its
//   own: about four pairs per sample, where a thread per leaf used to test
//   every sample and add its shares as it went.  Every sample is tested
//   against every leaf, without divergence and eight operations each.
// The tree lives in shared memory while it is small enough.  Its rectangles,
// the bottom-up weights and the new tree's depth-first numbering run level by
// level over a breadth-first list: a node's children come after those of every
// node that splits before it in depth-first order, a prefix of the subtrees'
// split counts (one thread walked the tree in global memory before).
// Latency bound: a block per region, so few regions leave SMs idle.  First fit of
// 786,432 + 262,144 samples in 48 regions 21.3 -> 2.3 ms, the next Update of 96
// regions 1.8 -> 0.75 ms (about 200 leaves and four pairs per sample).
#include <cuda_runtime.h>

#include <cstdint>

#include "dqt.cuh"
#include "launch.h"
#include "pgl_internal.h"

namespace pgl {

constexpr int kDqtThreads = 512;
constexpr uint32_t kDqtNodes = 768;      // trees up to this many nodes are held in shared memory
constexpr uint32_t kDqtPool = 10240;     // words for the shares and the masks of a chunk
// Two Updates of 200,000 samples in regions of 16,000, us, by leaves whose rectangles are held
// in shared memory / leaves of a sample that a thread keeps / leaves up to which a chunk's
// shares are a matrix (the others at their values below):
//                                 rects 128  256  512   list 8   16   32   matrix 0   20   40   80
//   default arguments                  1700 1650 1640     1630 1640 1660     1820 1640 1640 1790
//   threshold 0.1, 6 levels            1870 1890 1880     1880 1880 1880     2300 1990 1880 1870
//   threshold 0.002                    2630 2630 2540     2550 2540 2540     2790 2540 2540 2720
//   threshold 0.02                     2200 2200 2190     2140 2190 2360     2450 2200 2190 2340
//   footprint 4                        6990 6910 6900     6890 6900 6920     9860 6890 6900 5060
// (more leaves in the matrix mean fewer samples per chunk: the wide boxes of the last row gain,
// the ordinary ones lose.)
constexpr uint32_t kDqtRects = 512, kDqtList = 16, kDqtDense = 40;
constexpr int kDqtLevels = 40;           // levels of a tree at most

struct DqtShared {
  __align__(16) float pool[kDqtPool];
  __align__(16) float ones[kDqtThreads + 8];
  __align__(16) float first[kDqtThreads + 8], second[kDqtThreads + 8];
  float4 box[kDqtThreads];
  float4 leafRect[kDqtRects];
  float area[kDqtThreads];
  DqtStatsNode stats[kDqtNodes];
  Box2 rect[kDqtNodes];
  uint32_t order[kDqtNodes], count[kDqtNodes], base[kDqtNodes], newIndex[kDqtNodes];
  uint32_t levelAt[kDqtLevels + 2];
  uint32_t warpSum[kDqtThreads / 32];
  uint32_t numLeaves, tail;
  uint16_t longs[kDqtThreads];  // threads of the chunk that found more leaves than that
  uint32_t numLongs;
  int over;
};

// the statistics' decay (Statistics::decay, DQTFactory.h:109-116)
__device__ void dqt_decay(DqtHead &h, DqtStatsNode *S, float a) {
  if (threadIdx.x == 0) h.numSamples *= a;
  for (uint32_t i = threadIdx.x; i < h.numNodes; i += blockDim.x) {
    S[i].numSamples *= a;
    S[i].first *= a;
    S[i].second *= a;
  }
  __syncthreads();
}

struct DqtScratch {  // per block, `scratchStride` entries each: trees too large for shared memory
  Box2 *rect;
  float4 *leafRect;
  DqtStatsNode *build;
  uint32_t *order, *count, *base, *newIndex;
};

__device__ __noinline__ float dqt_divide(float a, float b) { return a / b; }
// a leaf's share a / area of a box, area not 0; y = RN(1 / area), 0 where the division is needed
__device__ __forceinline__ float dqt_share(float a, float area, float y) {
  if (y == 0.0f || (a < 1e-25f && a != 0.0f)) return dqt_divide(a, area);
  return markstein_q(a, area, y);
}
__device__ __forceinline__ float dqt_overlap(float4 f, float4 r) {
  return Box2{f.x, f.y, f.z, f.w}.intersect(Box2{r.x, r.y, r.z, r.w}).area();
}

// One update of a region's statistics and quadtree with `n` samples; `points`
// keeps their points on the square and moments (written unless `mapped`).
__device__ void dqt_update(DqtShared &X, DqtHead &h, DqtStatsNode *Sg, DqtNode *N, uint32_t stride,
                           const DqtScratch &Y, const float4 *dirw, const float *pdf, float4 *points, bool mapped,
                           uint32_t n, const DqtArgs &cfg, int *err) {
  // the factory's dispatch runs no branch for other values (DQTFactory.h:168-185)
  if (!(cfg.footprintFactor >= 0.0f) || (cfg.leafEstimator != 0 && cfg.leafEstimator != 1) ||
      (cfg.splitMetric != 0 && cfg.splitMetric != 1))
    return;
  const float ff = cfg.footprintFactor;
  const uint32_t tid = threadIdx.x, numNodes = h.numNodes;
  const bool small = numNodes <= kDqtNodes;
  DqtStatsNode *S = small ? X.stats : Sg;
  Box2 *rect = small ? X.rect : Y.rect;
  uint32_t *order = small ? X.order : Y.order, *count = small ? X.count : Y.count;
  uint32_t *base = small ? X.base : Y.base, *newIndex = small ? X.newIndex : Y.newIndex;
  if (small)
    for (uint32_t i = tid; i < numNodes; i += kDqtThreads) S[i] = Sg[i];
  if (tid == 0) {
    h.numSamples += float(n);
    rect[0] = Box2{0.f, 0.f, 1.f, 1.f};
    order[0] = 0;
    X.levelAt[0] = 0;
    X.tail = 1;
    X.numLeaves = 0;
    X.over = 0;
  }
  __syncthreads();
  // the nodes by level, their rectangles, and the leaves (their numbers in
  // `count`, their nodes in `base`)
  int levels = 0;
  for (uint32_t from = 0;; ++levels) {
    const uint32_t to = min(X.tail, numNodes);
    __syncthreads();
    if (tid == 0) X.levelAt[levels + 1] = to;
    if (to == from || levels >= kDqtLevels) break;
    for (uint32_t k = from + tid; k < to; k += kDqtThreads) {
      const uint32_t i = order[k], c0 = S[i].child;
      if (c0 > 0) {
        const uint32_t at = atomicAdd(&X.tail, 4u);
        const Box2 r = rect[i];
        for (uint32_t c = 0; c < 4 && at + c < numNodes; ++c) {  // a tree's nodes are all different
          order[at + c] = c0 + c;
          rect[c0 + c] = r.child(c);
        }
      } else {
        const uint32_t l = atomicAdd(&X.numLeaves, 1u);
        count[i] = l;
        base[l] = i;
      }
    }
    from = to;
    __syncthreads();
  }
  __syncthreads();
  const uint32_t L = X.numLeaves;
  float4 *leafRect = L <= kDqtRects ? X.leafRect : Y.leafRect;  // padded to a multiple of 32 with nothing
  for (uint32_t l = tid; l < ((L + 31) & ~31u); l += kDqtThreads) {
    // without a footprint a sample counts for the leaf that its point descends to, which may
    // have no width (its sides round together some 25 levels down): cells by number
    const Box2 cell{float(l), 0.f, float(l) + 1.f, 1.f};
    const Box2 r = l >= L ? Box2{2.f, 2.f, 1.f, 1.f} : ff > 0.0f ? rect[base[l]] : cell;
    leafRect[l] = make_float4(r.x0, r.y0, r.x1, r.y1);
  }
  // Samples per chunk: as many as the pool holds a matrix of shares for, or
  // masks, counts and at least five pairs per sample; with more leaves, masks
  // alone (the leaves' threads then compute the shares); beyond that (no
  // masks) they test every sample.
  const bool dense = ff > 0.0f && L <= kDqtDense;
  auto words32 = [&](uint32_t T) { return dense ? L * (T + 4) : L * (T / 32 + T / 64 + 7) + 15 * T; };
  uint32_t T = kDqtThreads;
  while (T > 64 && words32(T) > kDqtPool) T /= 2;
  const bool withSlots = !dense && words32(T) <= kDqtPool;
  if (!dense && !withSlots) {
    T = kDqtThreads;
    while (T > 32 && L * (T / 32) > kDqtPool) T /= 2;
  }
  const bool masks = !dense && L * (T / 32) <= kDqtPool;
  if (!dense && !masks) T = kDqtThreads;
  const uint32_t words = T / 32, row = T + 4;
  // the pool with slots: masks, pairs before each word of a leaf's (16 bits
  // each), first slot per leaf (multiples of four), then three rows of slots
  uint32_t *mask = reinterpret_cast<uint32_t *>(X.pool);
  uint16_t *before = reinterpret_cast<uint16_t *>(mask + L * words);
  uint32_t *slotOf = mask + L * words + (L * words + 1) / 2;
  const uint32_t used = (L * words + (L * words + 1) / 2 + L + 3) & ~3u;
  const uint32_t slots = withSlots ? ((kDqtPool - used) / 3) & ~3u : 0u;
  float *slot = X.pool + used;
  if (dense && tid < T) X.ones[tid] = 1.0f;
  // dense: thread c runs chain c / L (count, first, second moment) of leaf c % L
  const bool chain = dense && tid < 3 * L;
  const uint32_t chainLeaf = chain ? base[tid % L] : 0u, which = chain ? tid / L : 0u;
  float acc = 0.0f;
  if (chain) acc = which == 0 ? S[chainLeaf].numSamples : which == 1 ? S[chainLeaf].first : S[chainLeaf].second;
  __syncthreads();
  for (uint32_t at = 0; at < n; at += T) {
    const uint32_t cnt = min(T, n - at);
    if (tid < cnt) {
      float px, py, first, second;
      if (mapped) {
        const float4 pt = points[at + tid];
        px = pt.x;
        py = pt.y;
        first = pt.z;
        second = pt.w;
      } else {
        const float4 d = dirw[at + tid];
        const float p = pdf[at + tid];
        if (cfg.leafEstimator == 0) {  // REJECTION_SAMPLING
          first = d.w;
          second = d.w * d.w * p;
        } else {  // PER_LEAF
          first = d.w * p;
          second = first * first;
        }
        dqt_dir_to_point(d.x, d.y, d.z, px, py);
        points[at + tid] = make_float4(px, py, first, second);
      }
      Box2 leaf;
      const uint32_t li = dqt_query(S, px, py, leaf);
      const float cell = float(count[li]);
      Box2 filter{cell, 0.f, cell + 1.f, 1.f};
      float area = 1.0f;
      if (ff > 0.0f) {
        const float hx = ff * (leaf.x1 - leaf.x0) / 2.0f, hy = ff * (leaf.y1 - leaf.y0) / 2.0f;
        filter = Box2{px - hx, py - hy, px + hx, py + hy}.intersect(Box2{0.f, 0.f, 1.f, 1.f});
        area = filter.area();
        if (area == 0.0f) area = 1.0f;  // its sides round to the point: it overlaps nothing and gives no shares
      }
      X.box[tid] = make_float4(filter.x0, filter.y0, filter.x1, filter.y1);
      X.area[tid] = area;
      X.first[tid] = first;
      X.second[tid] = second;
    } else if (tid < T) {
      X.box[tid] = make_float4(2.f, 2.f, 1.f, 1.f);  // overlaps nothing
      X.area[tid] = 1.0f;
    }
    if (tid == 0) X.numLongs = 0;
    __syncthreads();
    // thread (part, sample): its part of the leaves (a point on the square is never NaN)
    const uint32_t s = tid % T, part = tid / T, parts = kDqtThreads / T;
    const float4 box = X.box[s];
    const float area = X.area[s], inv = area >= 1e-25f && area <= 1e25f ? rcp_newton(area) : 0.0f;
    if (dense) {
      for (uint32_t l = part; l < L; l += parts) X.pool[l * row + s] = dqt_share(dqt_overlap(box, leafRect[l]), area, inv);
      __syncthreads();
      if (chain) {
        const float *w = X.pool + (tid % L) * row, *x = which == 0 ? X.ones : which == 1 ? X.first : X.second;
        for (uint32_t k = 0; k < cnt; k += 4) {  // past the chunk's last sample the shares are 0
          const float4 a = *reinterpret_cast<const float4 *>(w + k), b = *reinterpret_cast<const float4 *>(x + k);
          // a leaf that a sample does not overlap is left alone whatever the sample's value
          acc += a.x != 0.0f ? a.x * b.x : 0.0f;
          acc += a.y != 0.0f ? a.y * b.y : 0.0f;
          acc += a.z != 0.0f ? a.z * b.z : 0.0f;
          acc += a.w != 0.0f ? a.w * b.w : 0.0f;
        }
      }
      __syncthreads();
      continue;
    }
    uint32_t mine[kDqtList], found = 0;  // the sample's leaves of this part
    if (masks) {
      for (uint32_t g = part; g < (L + 31) / 32; g += parts) {  // 32 leaves at a time
        const float4 *R = leafRect + 32 * g;
        uint32_t hits = 0;
#pragma unroll
        for (uint32_t l = 0; l < 32; ++l) {
          const float4 r = R[l];
          // the overlap's area is zero exactly when one of its sides is
          if (fminf(box.z, r.z) > fmaxf(box.x, r.x) && fminf(box.w, r.w) > fmaxf(box.y, r.y)) hits |= 1u << l;
        }
        // bit l of lane s to bit s of lane l
        uint32_t m = 0x0000FFFFu, x = hits;
#pragma unroll
        for (uint32_t j = 16; j > 0; j >>= 1, m ^= m << j) {
          const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
          x = (tid & j) ? (x & ~m) | ((y >> j) & m) : (x & m) | ((y << j) & ~m);
        }
        if (32 * g + (tid & 31) < L) mask[(32 * g + (tid & 31)) * words + s / 32] = x;
        for (; hits != 0; hits &= hits - 1u) {
          if (found < kDqtList) mine[found] = 32 * g + uint32_t(__ffs(hits)) - 1u;
          ++found;
        }
      }
      if (found > kDqtList) {
        found = 0;
        X.longs[atomicAdd(&X.numLongs, 1u)] = uint16_t(tid);
      }
      __syncthreads();
    }
    uint32_t pairs = 0;
    if (withSlots) {
      // counts per leaf and word, then an exclusive sum over the leaves
      for (uint32_t k0 = 0; k0 < L; k0 += kDqtThreads) {
        const uint32_t k = k0 + tid;
        uint32_t c = 0;
        if (k < L)
          for (uint32_t q = 0; q < words; ++q) {
            before[k * words + q] = uint16_t(c);
            c += uint32_t(__popc(mask[k * words + q]));
          }
        c = (c + 3u) & ~3u;
        uint32_t sum = c;
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, sum, off);
          if ((tid & 31) >= uint32_t(off)) sum += o;
        }
        if ((tid & 31) == 31) X.warpSum[tid / 32] = sum;
        __syncthreads();
        uint32_t warpsBefore = 0, all = 0;
        for (uint32_t q = 0; q < kDqtThreads / 32; ++q) {
          warpsBefore += q < tid / 32 ? X.warpSum[q] : 0u;
          all += X.warpSum[q];
        }
        if (k < L) slotOf[k] = pairs + warpsBefore + sum - c;
        pairs += all;
        __syncthreads();
      }
    }
    if (withSlots && pairs <= slots) {  // nearly always
      auto put = [&](uint32_t l, uint32_t t, float w) {
        const uint32_t m = mask[l * words + t / 32], e = slotOf[l] + before[l * words + t / 32] +
                                                         uint32_t(__popc(m & ((1u << (t & 31)) - 1u)));
        slot[e] = w;  // without a share the sample's moments do not count, whatever they are
        slot[slots + e] = w != 0.0f ? w * X.first[t] : 0.0f;
        slot[2 * slots + e] = w != 0.0f ? w * X.second[t] : 0.0f;
      };
      for (uint32_t j = 0; j < found; ++j)
        put(mine[j], s, ff > 0.0f ? dqt_share(dqt_overlap(box, leafRect[mine[j]]), area, inv) : 1.0f);
      for (uint32_t q = tid / 32; q < X.numLongs; q += kDqtThreads / 32) {  // a warp for a long list
        const uint32_t t = X.longs[q] % T;
        for (uint32_t k = 32 * (X.longs[q] / T) + (tid & 31); k < L; k += 32 * parts)
          if (mask[k * words + t / 32] >> (t & 31) & 1u) put(k, t, dqt_share(dqt_overlap(X.box[t], leafRect[k]), X.area[t], 0.0f));
      }
      for (uint32_t k = tid; k < L; k += kDqtThreads) {  // the slots that round a leaf's up to a multiple of four
        const uint32_t q = k * words + words - 1;
        const uint32_t c = before[q] + uint32_t(__popc(mask[q]));
        for (uint32_t e = slotOf[k] + c; e < slotOf[k] + ((c + 3u) & ~3u); ++e)
          slot[e] = slot[slots + e] = slot[2 * slots + e] = 0.0f;
      }
      __syncthreads();
      for (uint32_t k = tid; k < L; k += kDqtThreads) {
        const uint32_t from = slotOf[k], to = k + 1 < L ? slotOf[k + 1] : pairs;
        if (from == to) continue;
        DqtStatsNode &node = S[base[k]];
        float ns = node.numSamples, fs = node.first, ss = node.second;
        const float4 *u = reinterpret_cast<const float4 *>(slot), *v = reinterpret_cast<const float4 *>(slot + slots),
                     *w = reinterpret_cast<const float4 *>(slot + 2 * slots);
#pragma unroll 2
        for (uint32_t e = from / 4; e < to / 4; ++e) {
          const float4 a = u[e], b = v[e], c = w[e];
          ns += a.x;
          fs += b.x;
          ss += c.x;
          ns += a.y;
          fs += b.y;
          ss += c.y;
          ns += a.z;
          fs += b.z;
          ss += c.z;
          ns += a.w;
          fs += b.w;
          ss += c.w;
        }
        node.numSamples = ns;
        node.first = fs;
        node.second = ss;
      }
    } else {
      for (uint32_t k = tid; k < L; k += kDqtThreads) {
        const float4 r = leafRect[k];
        DqtStatsNode &node = S[base[k]];
        float ns = node.numSamples, fs = node.first, ss = node.second;
        auto add = [&](uint32_t t) {
          float w = dqt_overlap(X.box[t], r);
          if (w == 0.0f) return;
          w = ff > 0.0f ? w / X.area[t] : 1.0f;
          ns += w;
          fs += w * X.first[t];
          ss += w * X.second[t];
        };
        if (masks) {
          for (uint32_t q = 0; q < words; ++q)
            for (uint32_t bits = mask[k * words + q]; bits != 0; bits &= bits - 1u) add(32 * q + uint32_t(__ffs(bits)) - 1u);
        } else {
          for (uint32_t t = 0; t < cnt; ++t) add(t);
        }
        node.numSamples = ns;
        node.first = fs;
        node.second = ss;
      }
    }
    __syncthreads();
  }
  if (chain) {
    if (which == 0) S[chainLeaf].numSamples = acc;
    else if (which == 1) S[chainLeaf].first = acc;
    else S[chainLeaf].second = acc;
  }
  __syncthreads();
  // sample and split weights bottom-up (DQTFactory.h:232-263)
  for (uint32_t k = tid; k < L; k += kDqtThreads) {
    const uint32_t i = base[k];
    DqtStatsNode &m = S[i];
    const float f = cfg.leafEstimator == 0 ? 1.0f / h.numSamples : dqt_area(rect[i]) / m.numSamples;
    const float first = m.first * f, second = m.second * f;
    m.sampleWeight = first;
    m.splitWeight = cfg.splitMetric == 0 ? first : sqrtf(dqt_area(rect[i]) * second);
  }
  __syncthreads();
  for (int v = levels - 1; v >= 0; --v) {
    for (uint32_t k = X.levelAt[v] + tid; k < X.levelAt[v + 1]; k += kDqtThreads) {
      DqtStatsNode &m = S[order[k]];
      if (m.child == 0) continue;
      float sample = 0.0f, split = 0.0f;
      for (uint32_t c = 0; c < 4; ++c) {
        sample += S[m.child + c].sampleWeight;
        split += S[m.child + c].splitWeight;
      }
      m.sampleWeight = sample;
      m.splitWeight = split;
    }
    __syncthreads();
  }
  // buildRecursive (DQTFactory.h:283-311): the new tree in depth-first order, a
  // node's four children allocated together when it is reached.  Bottom-up the
  // nodes that split in each node's part of the new tree, top-down the splits
  // before it; a leaf that splits gives its children a quarter of its
  // statistics (DQTFactory.h:313-324).
  const float limit = cfg.splitThreshold * S[0].splitWeight;
  for (int v = levels - 1; v >= 0; --v) {
    for (uint32_t k = X.levelAt[v] + tid; k < X.levelAt[v + 1]; k += kDqtThreads) {
      const uint32_t i = order[k], c0 = S[i].child;
      uint32_t splits = 0;
      if (uint32_t(v) < cfg.maxLevels && S[i].splitWeight > limit) {
        splits = 1;
        if (c0 > 0)
          for (uint32_t c = 0; c < 4; ++c) splits += count[c0 + c];
        if (v + 1 >= kDqtLevels) X.over = 1;
      }
      count[i] = splits;
      newIndex[i] = ~0u;
    }
    __syncthreads();
  }
  // a tree over the node bound (not possible for the bound's arguments)
  // keeps its previous nodes and fails the launch
  const uint32_t size = 1u + 4u * count[0];
  const bool over = size > stride || X.over != 0;
  if (tid == 0) {
    newIndex[0] = 0;
    base[0] = 0;
    if (over) atomicCAS(err, 0, 3);
  }
  __syncthreads();
  if (over) return;
  for (int v = 0; v < levels; ++v) {
    for (uint32_t k = X.levelAt[v] + tid; k < X.levelAt[v + 1]; k += kDqtThreads) {
      const uint32_t i = order[k], j = newIndex[i];
      if (j == ~0u) continue;
      DqtStatsNode on = S[i];
      const uint32_t old = on.child, c0 = 1u + 4u * base[i];
      on.child = count[i] > 0 ? c0 : 0u;
      Y.build[j] = on;
      if (count[i] == 0) continue;
      if (old > 0) {
        uint32_t b = base[i] + 1u;
        for (uint32_t c = 0; c < 4; ++c) {
          newIndex[old + c] = c0 + c;
          base[old + c] = b;
          b += count[old + c];
        }
      } else {
        const DqtStatsNode part{0u, on.sampleWeight / 4, on.splitWeight / 4, on.numSamples / 4, on.first / 4,
                                on.second / 4};
        for (uint32_t c = 0; c < 4; ++c) Y.build[c0 + c] = part;
      }
    }
    __syncthreads();
  }
  for (uint32_t i = tid; i < size; i += kDqtThreads) {
    const DqtStatsNode b = Y.build[i];
    Sg[i] = b;
    N[i] = DqtNode{b.child, b.sampleWeight};
  }
  if (tid == 0) h.numNodes = size;
  __syncthreads();
}

__device__ bool dqt_stats_ok(float v) { return !isnan(v) && !isinf(v) && v >= 0.0f; }

__global__ void __launch_bounds__(kDqtThreads)
dqt_update_kernel(const LeafTask *tasks, uint32_t numTasks, unsigned int *queue, DqtSides sides, Box2 *rects,
                  DqtStatsNode *builds, uint32_t *leaves, uint32_t scratchStride, int *err) {
  extern __shared__ __align__(16) unsigned char dqt_smem[];
  DqtShared &X = *reinterpret_cast<DqtShared *>(dqt_smem);
  __shared__ uint32_t taskId;
  __shared__ uint32_t statsBad;
  uint32_t *words = leaves + size_t(blockIdx.x) * 4 * scratchStride;
  Box2 *rect = rects + size_t(blockIdx.x) * 2 * scratchStride;
  const DqtScratch Y{rect, reinterpret_cast<float4 *>(rect + scratchStride), builds + size_t(blockIdx.x) * scratchStride,
                     words, words + scratchStride, words + 2 * size_t(scratchStride), words + 3 * size_t(scratchStride)};
  for (;;) {
    if (threadIdx.x == 0) taskId = atomicAdd(queue, 1u);
    __syncthreads();
    if (taskId >= numTasks) break;
    const LeafTask t = tasks[taskId];
    const DqtSide &D = sides.side[(t.flags & kTaskVolume) ? 1 : 0];
    DqtHead &h = D.heads[t.region];
    DqtStatsNode *S = D.stats + size_t(t.region) * D.stride;
    DqtNode *N = D.nodes + size_t(t.region) * D.stride;
    const bool fit = (t.flags & kTaskFit) != 0;
    if (fit) {
      if (t.count > 0) {  // fitRegions (Field.h:389-439 -> DQTFactory.h:149-155): five decayed passes
        for (int k = 0; k < 5; ++k) {
          dqt_decay(h, S, 0.25f);
          dqt_update(X, h, S, N, D.stride, Y, D.dirw + t.begin, D.pdf + t.begin, D.points + t.begin, k > 0, t.count, D.args, err);
        }
        if (threadIdx.x == 0) {
          h.pivot[0] = t.mean[0];
          h.pivot[1] = t.mean[1];
          h.pivot[2] = t.mean[2];
          h.valid = (!isinf(N[0].weight) && N[0].weight > 0.0f) ? 1u : 0u;
        }
      } else if (threadIdx.x == 0) {
        h.valid = 0;
      }
    } else {
      if (t.flags & kTaskDecay) dqt_decay(h, S, D.decay);  // Field.h:457-461
      if (t.count > 0) {
        dqt_update(X, h, S, N, D.stride, Y, D.dirw + t.begin, D.pdf + t.begin, D.points + t.begin, false, t.count, D.args, err);
        // DirectionalQuadtree::isValid and Statistics::isValid (DQT.h:40-42, DQTFactory.h:95-107)
        if (threadIdx.x == 0) statsBad = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < h.numNodes; i += blockDim.x) {
          const DqtStatsNode &m = S[i];
          if (!dqt_stats_ok(m.sampleWeight) || !dqt_stats_ok(m.splitWeight) || !dqt_stats_ok(m.numSamples) ||
              !dqt_stats_ok(m.first) || !dqt_stats_ok(m.second))
            atomicOr(&statsBad, 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          const bool treeOk = !isinf(N[0].weight) && N[0].weight > 0.0f;
          const bool statsOk = !statsBad && S[0].sampleWeight > 0.0f && S[0].splitWeight > 0.0f;
          h.valid = (treeOk && statsOk) ? 1u : 0u;
        }
      }
    }
    __syncthreads();
  }
}

// New regions start as copies of the region they split from (head and both
// node arrays).
__global__ void dqt_copy_kernel(DqtHead *heads, DqtStatsNode *stats, DqtNode *nodes, uint32_t stride,
                                const uint32_t *dst, const uint32_t *src, uint32_t n) {
  const uint32_t k = blockIdx.x;
  if (k >= n) return;
  const uint32_t a = src[k], b = dst[k];
  if (threadIdx.x == 0) heads[b] = heads[a];
  const uint32_t m = heads[a].numNodes;
  for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
    stats[size_t(b) * stride + i] = stats[size_t(a) * stride + i];
    nodes[size_t(b) * stride + i] = nodes[size_t(a) * stride + i];
  }
}

// A region in the reference's initial state: one leaf, zero statistics.
__global__ void dqt_init_kernel(DqtHead *heads, DqtStatsNode *stats, DqtNode *nodes, uint32_t stride, uint32_t first,
                                uint32_t n) {
  const uint32_t r = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= first + n) return;
  heads[r] = DqtHead{{0.f, 0.f, 0.f}, 0.0f, 1u, 0u, {0u, 0u}};
  stats[size_t(r) * stride] = DqtStatsNode{0u, 0.f, 0.f, 0.f, 0.f, 0.f};
  nodes[size_t(r) * stride] = DqtNode{0u, 0.f};
}

cudaError_t launch_dqt_update(const LeafTask *tasks, uint32_t numTasks, unsigned int *queue, const DqtSides &sides,
                              Box2 *rects, DqtStatsNode *builds, uint32_t *leaves, uint32_t scratchStride, int blocks,
                              int *err, cudaStream_t s) {
  if (numTasks == 0) return cudaSuccess;
  // once per process (thread-safe static initialisation)
  static const cudaError_t attr =
      cudaFuncSetAttribute(dqt_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(DqtShared)));
  if (attr != cudaSuccess) return attr;
  count_launch();
  dqt_update_kernel<<<unsigned(blocks), kDqtThreads, sizeof(DqtShared), s>>>(tasks, numTasks, queue, sides, rects, builds, leaves,
                                                             scratchStride, err);
  return cudaGetLastError();
}
cudaError_t launch_dqt_copy(DqtHead *heads, DqtStatsNode *stats, DqtNode *nodes, uint32_t stride, const uint32_t *dst,
                            const uint32_t *src, uint32_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  dqt_copy_kernel<<<n, 256, 0, s>>>(heads, stats, nodes, stride, dst, src, n);
  return cudaGetLastError();
}
cudaError_t launch_dqt_init(DqtHead *heads, DqtStatsNode *stats, DqtNode *nodes, uint32_t stride, uint32_t first,
                            uint32_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  count_launch();
  dqt_init_kernel<<<(n + 127) / 128, 128, 0, s>>>(heads, stats, nodes, stride, first, n);
  return cudaGetLastError();
}

}  // namespace pgl
