// Per-leaf directional fitting on the GPU: parallax-aware vMF mixtures fitted
// by weighted MAP-EM with chi-square split and merge, one thread block per
// leaf (region), leaves handed out by an atomic work queue.
//
// What it computes is Open PGL's AdaptiveSplitAndMergeFactory::fit/update
// (directional/vmm/AdaptiveSplitandMergeFactory.h:303-462) on a leaf's
// deterministically sorted, parallax-reprojected samples, with the weighted EM
// of ParallaxAwareVonMisesFisherWeightedEMFactory.h:717-1326 and the splitter
// and merger of VMMChiSquareComponentSplitter.h / VMMChiSquareComponentMerger.h.
//
// How it is laid out for the GPU: a pass over a leaf's samples (E-step,
// distance pass, split-statistics pass) streams the samples in chunks through
// a two-stage producer/consumer pipeline (see "sample passes" below):
// producer threads compute each sample's lobe terms and pdf, consumer threads
// (one per accumulator, e.g. the x component of lobe 7's weighted direction
// sum) add the chunk's terms in sample order.  That keeps the reference's
// summation order (sequential over samples within each SIMD lane), so every
// accumulator gets the reference's bits.  Per-leaf logic between the passes runs
// on one warp, a lane per lobe (M step, splits, shifts, checks), on the whole block
// (merge costs) or on thread 0.
#include <cuda_runtime.h>

#include <cstddef>

#include "launch.h"
#include "pgl_internal.h"

namespace pgl {

constexpr int kEmThreads = 512;
constexpr int kStageFloats = 19968;  // floats per pipeline stage (two stages, 156 KB)

// E-step passes shared between blocks.  Every block owns a board and a ring of
// chunk slots in global memory.  For each E-step pass the home block publishes
// the pass on its board (lobe parameters, sample range, chunk shape).  Its own
// producer warps take chunks from the board's grab word and write them
// straight into its shared-memory stages; a block that has run out of leaves
// (a helper) takes chunks from the same grab word and writes them into the
// ring, from where the home block's loader warp copies them into the stages
// with bulk copies.  The consumer warps add the chunks in chunk order.
constexpr int kMaxStages = 8;                          // consumer pipeline stages
constexpr int kMaxChunk = 416;                         // E-step samples per chunk at most (13 producer warps)
constexpr uint32_t kRingFloats = 65536;                // ring per block (256 KB)
constexpr uint32_t kRingMaxSlots = 64;
constexpr unsigned long long kWaitNs = 2000000000ull;  // longest wait before the launch fails
constexpr uint32_t kGrabIdxBits = 22;                  // grab word: generation | chunks | next chunk
constexpr uint32_t kGrabMask = (1u << kGrabIdxBits) - 1u;
constexpr uint32_t kGrabGenMask = (1u << 20) - 1u;
constexpr uint32_t kMaxSharedChunks = kGrabMask - 4096u;

// Lobe parameters by pairs: entry pair_at(k) + c, three entries per pair of
// lobes and one of padding per lobe vector, so that lanes on different vectors
// read distinct banks.
constexpr int kPairEntries = (3 * kLanes / 2 + 1) * (kMaxK / kLanes);
__host__ __device__ constexpr int pair_at(int k) { return (k / kLanes) * (3 * kLanes / 2 + 1) + 3 * ((k % kLanes) / 2); }

enum EmError { kErrNone = 0, kErrChunkWait = 1, kErrSlotWait = 2, kErrCopyWait = 3, kErrLeafTooLarge = 4 };

struct __align__(16) BoardParams {  // one pass as its home block publishes it
  float4 lobeP[kPairEntries];
  const float4 *dirw;
  uint32_t count, seqBase, cnt, pad;
};
struct __align__(128) Board {
  unsigned long long grab;     // generation (bits 44..63), chunks (22..43), next chunk (0..21)
  uint32_t pad0[30];
  uint32_t consumed;           // chunks (sequence numbers) whose ring slots are free again
  uint32_t pad1[31];
  uint32_t helpers;            // helper blocks attached to the board (at most EmTuning::maxHelpers)
  uint32_t pad2[31];
  uint32_t ready[kRingMaxSlots];  // per ring slot: sequence number of the chunk it holds
  BoardParams params[2];          // by generation parity
};

struct Unassigned {
  float sw, dx, dy, dz;
};

constexpr int kMergePairs = 256;  // merge costs computed at once
struct MergeParts {               // see merge_costs
  float mx[kMergePairs], my[kMergePairs], mz[kMergePairs], kappa[kMergePairs], norm[kMergePairs], e2k[kMergePairs];
  // products of pairs, then of the components with themselves
  float px[kMergePairs + kMaxK], py[kMergePairs + kMaxK], pz[kMergePairs + kMaxK], pkappa[kMergePairs + kMaxK],
      pnorm[kMergePairs + kMaxK], pscale[kMergePairs + kMaxK];
  float part[3][kMergePairs];
  uint8_t i[kMergePairs], j[kMergePairs];
};

struct EmShared {
  VMMState vmm;
  SuffState suff;     // training statistics ("previous" statistics of EM)
  SplitState split;   // training split statistics
  SuffState cur;      // statistics of the current EM iteration
  SuffState temp;     // statistics of a partial refit
  SplitState lsplit;  // split statistics used by the recursive splitting
  __align__(16) float pbuf[2 * kStageFloats];  // the two pipeline stages
  __align__(16) float4 lobeP[kPairEntries];   // see pack_pairs
  __align__(16) float4 frameP[kPairEntries];  // split passes: rows x and y of the lobes' inverse frames
  __align__(16) float ones[kMaxChunk + 48];  // the factor row of the chains that sum a_k w
  float2 lobeW[kMaxK];  // distance passes: weight, its reciprocal (0: divide)
  float xch[2][kMaxK];
  uint32_t rcpTab[2048];
  float cost[kMaxK][kMaxK];  // merge cost of components i < j (cost[i][j])
  MergeParts merge;
  float ll;
  Unassigned un;
  int mask[kMaxK];
  int loopFlag;
  int splitCount;
  int candIdx[kMaxK];
  float candChi[kMaxK];
  int numCands;
  float mcEstimate;
  int iterations;
  LeafReport report;
  LeafProfile prof;
  unsigned long long full[kMaxStages];  // stage holds its chunk (bulk copy or own producers)
  uint32_t stageUses[kMaxStages];       // completed phases of a stage's barrier
  uint32_t warpDone[kEmThreads / 32];   // chunks of the pass each consumer warp has added
  uint32_t own[64];    // sequence numbers of chunks this block's producers took
  BoardParams hp;      // a helper's copy of the pass it produces for
  Board *board;        // this block's board and ring
  float *ring;
  int *err;            // EmError of the launch
  uint32_t gen, seqBase, abortAt;
  EmTuning tune;       // the launch's schedule parameters (the same in every block)
  int hgrab[2], grabbed, helpBoard, helpExit;
  uint32_t grabGen;
  int grabExact;                                  // the chunk taken is the one whose slot was checked
  int nextGrabbed, nextExact, hasNext;            // a helper's next chunk, taken while producing
  uint32_t nextGen;
  uint32_t scanRem[kEmThreads / 32];
  int scanIdx[kEmThreads / 32];
};
static_assert(offsetof(EmShared, pbuf) % 16 == 0 && offsetof(EmShared, lobeP) % 16 == 0 &&
                  offsetof(EmShared, hp) % 16 == 0 && offsetof(EmShared, ones) % 16 == 0 && offsetof(EmShared, full) % 8 == 0,
              "128-bit shared loads");

// cycle accounting of thread 0 (LeafProfile)
#define PGL_PROF_BEGIN(t) const long long t = clock64();
#define PGL_PROF_END(t, field) \
  if (threadIdx.x == 0) S.prof.field += uint64_t(clock64() - (t));

// ---------------------------------------------------------------- scalar helpers (thread 0)

__device__ void vmm_calc_norm(VMMState &v) {  // PAVMM.h:852-863
  int c = vec_count(int(v.K));
  for (int k = 0; k < c * kLanes; ++k) {
    v.e2k[k] = fexp(-2.0f * v.kappa[k]);
    float nrm = v.kappa[k] / (kTwoPiF * (1.0f - v.e2k[k]));
    v.norm[k] = v.kappa[k] > 0.0f ? nrm : kInv4Pi;
  }
}
__device__ void vmm_calc_mean_cosines(VMMState &v) {  // PAVMM.h:866-877
  int c = vec_count(int(v.K));
  for (int k = 0; k < c * kLanes; ++k) {
    float th = 1.0f - 2.0f / (fexp(2.0f * v.kappa[k]) - 1.0f);
    float m = 1.0f / th - 1.0f / v.kappa[k];
    v.mc[k] = v.kappa[k] > 0.0f ? m : 0.0f;
  }
}
__device__ void vmm_init_uniform(VMMState &v, int K, float kappa, const float *dirs) {  // WEMFactory.h:633-664
  v.K = uint32_t(K);
  float weight = 1.0f / float(K);
  const float *d = dirs + (K - 1) * kMaxK * 3;
  for (int n = 0; n < kMaxK; ++n) {
    v.mx[n] = d[3 * n + 0];
    v.my[n] = d[3 * n + 1];
    v.mz[n] = d[3 * n + 2];
    if (n < K) {
      v.kappa[n] = kappa;
      v.w[n] = weight;
    } else {
      v.kappa[n] = 0.0f;
      v.w[n] = 0.0f;
      v.norm[n] = kInv4Pi;
      v.e2k[n] = 1.0f;
      v.mc[n] = 0.0f;
    }
  }
  vmm_calc_norm(v);
  vmm_calc_mean_cosines(v);
}
__device__ void vmm_swap(VMMState &v, int i, int j) {
  if (i == j) return;
#define PGL_SWAPF(a) { float t_ = v.a[i]; v.a[i] = v.a[j]; v.a[j] = t_; }
  PGL_SWAPF(w) PGL_SWAPF(kappa) PGL_SWAPF(e2k) PGL_SWAPF(mc) PGL_SWAPF(norm) PGL_SWAPF(mx) PGL_SWAPF(my) PGL_SWAPF(mz) PGL_SWAPF(dist)
#undef PGL_SWAPF
}
__device__ void vmm_clear(VMMState &v, int i) {
  v.w[i] = 0.0f; v.kappa[i] = 0.0f; v.e2k[i] = 1.0f; v.mc[i] = 0.0f; v.norm[i] = kInv4Pi;
  v.mx[i] = 0.0f; v.my[i] = 0.0f; v.mz[i] = 1.0f; v.dist[i] = 0.0f;
}
__device__ void vmm_merge(VMMState &v, int i0, int i1) {  // PAVMM.h:259-343
  if (i0 == i1) return;
  float w0 = v.w[i0], w1 = v.w[i1], mc0 = v.mc[i0], mc1 = v.mc[i1];
  float kappa = 0.0f, nrm = kInv4Pi, e2k = 1.0f, w = w0 + w1;
  float mx = (w0 * mc0) * v.mx[i0] + (w1 * mc1) * v.mx[i1];
  float my = (w0 * mc0) * v.my[i0] + (w1 * mc1) * v.my[i1];
  float mz = (w0 * mc0) * v.mz[i0] + (w1 * mc1) * v.mz[i1];
  mx /= w; my /= w; mz /= w;
  float mc = mx * mx + my * my + mz * mz;
  if (mc > 0.0f) {
    mc = sqrtf(mc);
    kappa = mean_cosine_to_kappa(mc);
    kappa = kappa < 1e-3f ? 0.f : kappa;
    e2k = lib_expf(-2.0f * kappa);
    nrm = vmf_norm_double(kappa, e2k);
    mx /= mc; my /= mc; mz /= mc;
  } else {
    mx = v.mx[i0]; my = v.my[i0]; mz = v.mz[i0];
  }
  v.w[i0] = w; v.kappa[i0] = kappa; v.mc[i0] = mc; v.norm[i0] = nrm; v.e2k[i0] = e2k;
  v.mx[i0] = mx; v.my[i0] = my; v.mz[i0] = mz;
  float nd = w0 * v.dist[i0] + w1 * v.dist[i1];
  nd /= (w0 + w1);
  v.dist[i0] = nd;
  vmm_swap(v, i1, int(v.K) - 1);
  vmm_clear(v, int(v.K) - 1);
  v.K -= 1;
}
// The two lobes of a split (PAVMM.h:225-255); the caller sets K and the norms.
__device__ void vmm_split(VMMState &v, int i0, int i1, float w0, float w1, V3 m0, V3 m1, float mc0, float mc1) {
  v.dist[i1] = v.dist[i0];
  v.w[i0] = w0; v.mc[i0] = mc0; v.kappa[i0] = mean_cosine_to_kappa(mc0);
  v.mx[i0] = m0.x; v.my[i0] = m0.y; v.mz[i0] = m0.z;
  v.w[i1] = w1; v.mc[i1] = mc1; v.kappa[i1] = mean_cosine_to_kappa(mc1);
  v.mx[i1] = m1.x; v.my[i1] = m1.y; v.mz[i1] = m1.z;
}
__device__ void vmm_parallax_shift(VMMState &v, V3 s, int k) {  // PAVMM.h:809-831, lobe k; the caller moves the pivot
  V3 p = mk(v.mx[k], v.my[k], v.mz[k]) * v.dist[k] + s;
  float len = length(p);
  p = p / len;
  bool cond = (v.dist[k] > 0.0f) && (v.dist[k] >= -FLT_MAX) && (v.dist[k] <= FLT_MAX);
  if (cond) { v.mx[k] = p.x; v.my[k] = p.y; v.mz[k] = p.z; }
  v.dist[k] = v.dist[k] > 0.0f ? len : 0.0f;
}
// Validity of a region's state: one warp, a lane per lobe.
__device__ bool vmm_is_valid(const VMMState &v) {  // PAVMM.h:422-513
  const uint32_t k = threadIdx.x & 31;
  bool ok;
  if (k < v.K) {
    ok = isvalidf(v.w[k]) && v.w[k] >= 0.0f && v.w[k] <= 1.0f + 1e-6f;
    ok = ok && isvalidf(v.kappa[k]) && v.kappa[k] >= 0.0f;
    ok = ok && isvalidf(v.mc[k]) && v.mc[k] >= 0.0f && v.mc[k] <= 1.0f;
    ok = ok && isvalidf(v.mx[k]) && v.mx[k] >= -1.0f && v.mx[k] <= 1.0f;
    ok = ok && isvalidf(v.my[k]) && v.my[k] >= -1.0f && v.my[k] <= 1.0f;
    ok = ok && isvalidf(v.mz[k]) && v.mz[k] >= -1.0f && v.mz[k] <= 1.0f;
    ok = ok && isvalidf(v.norm[k]) && v.norm[k] >= 0.0f && isvalidf(v.e2k[k]);
    ok = ok && isvalidf(v.dist[k]) && v.dist[k] >= 0.0f;
  } else {
    ok = v.w[k] == 0.0f && v.kappa[k] == 0.0f && v.mx[k] == 0.0f && v.my[k] == 0.0f && v.mz[k] == 1.0f;
    ok = ok && v.mc[k] == 0.0f && fabsf(v.norm[k] - kInv4Pi) < 1e-6f && v.e2k[k] == 1.0f && v.dist[k] == 0.0f;
  }
  return __all_sync(0xFFFFFFFFu, ok);
}

__device__ void suff_clear(SuffState &s, uint32_t K) {
  s.K = K;
  int c = vec_count(int(K));
  for (int k = 0; k < c * kLanes; ++k) s.dx[k] = s.dy[k] = s.dz[k] = s.w[k] = s.dw[k] = 0.0f;
  s.sumWeights = 0.0f; s.numSamples = 0.0f; s.normalized = 0;
}
__device__ void suff_add(SuffState &a, const SuffState &b) {  // WEMFactory.h:575-593
  int c = vec_count(int(a.K));
  a.sumWeights += b.sumWeights;
  a.numSamples += b.numSamples;
  a.overallNumSamples += b.numSamples;
  for (int k = 0; k < c * kLanes; ++k) {
    a.dx[k] += b.dx[k]; a.dy[k] += b.dy[k]; a.dz[k] += b.dz[k]; a.w[k] += b.w[k]; a.dw[k] += b.dw[k];
  }
}
__device__ void suff_masked_replace(SuffState &a, const int *mask, const SuffState &b) {  // WEMFactory.h:448-468
  float sv[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int k = 0; k < kMaxK; ++k) {
    if (mask[k]) { a.dx[k] = b.dx[k]; a.dy[k] = b.dy[k]; a.dz[k] = b.dz[k]; a.w[k] = b.w[k]; a.dw[k] = b.dw[k]; }
    sv[k % kLanes] += a.w[k];
  }
  if (a.normalized) a.numSamples = reduce8(sv); else a.sumWeights = reduce8(sv);
}
__device__ void suff_decay(SuffState &s, float a) {
  for (int k = 0; k < kMaxK; ++k) { s.dx[k] *= a; s.dy[k] *= a; s.dz[k] *= a; s.w[k] *= a; s.dw[k] *= a; }
  s.numSamples *= a; s.sumWeights *= a;
}
__device__ void suff_parallax_shift(SuffState &s, const VMMState &v, V3 shift, int k) {  // WEMFactory.h:265-283, lobe k
  V3 d0 = mk(s.dx[k], s.dy[k], s.dz[k]);
  float smc = length(d0);
  V3 d = d0 / smc;
  d = d * v.dist[k];
  d = d + shift;
  d = d / length(d);
  d = d * smc;
  d = smc > 0.0f ? d : d0;
  if (v.dist[k] > 0.0f) { s.dx[k] = d.x; s.dy[k] = d.y; s.dz[k] = d.z; }
}
__device__ void suff_split(SuffState &s, int i, int j, V3 m0, V3 m1, float mc0, float mc1) {  // WEMFactory.h:516-550
  float sw = s.w[i];
  sw /= 2.0f;
  s.w[i] = sw; s.dx[i] = (m0.x * mc0) * sw; s.dy[i] = (m0.y * mc0) * sw; s.dz[i] = (m0.z * mc0) * sw;
  s.w[j] = sw; s.dx[j] = (m1.x * mc1) * sw; s.dy[j] = (m1.y * mc1) * sw; s.dz[j] = (m1.z * mc1) * sw;
  float t = s.dw[i] * 0.5f;
  s.dw[i] = t; s.dw[j] = t;
}
__device__ void suff_merge(SuffState &s, int i0, int i1) {  // WEMFactory.h:485-513
  int L = int(s.K) - 1;
  s.dx[i0] += s.dx[i1]; s.dy[i0] += s.dy[i1]; s.dz[i0] += s.dz[i1]; s.w[i0] += s.w[i1]; s.dw[i0] += s.dw[i1];
  s.dx[i1] = s.dx[L]; s.dy[i1] = s.dy[L]; s.dz[i1] = s.dz[L]; s.w[i1] = s.w[L]; s.dw[i1] = s.dw[L];
  s.dx[L] = s.dy[L] = s.dz[L] = s.w[L] = s.dw[L] = 0.0f;
  s.K--;
}
__device__ bool suff_is_valid(const SuffState &s) {
  const uint32_t k = threadIdx.x & 31;
  const bool ok = k < s.K ? isvalidf(s.dx[k]) && isvalidf(s.dy[k]) && isvalidf(s.dz[k]) && isvalidf(s.w[k]) &&
                                s.w[k] >= 0.0f && isvalidf(s.dw[k]) && s.dw[k] >= 0.0f
                          : s.dx[k] == 0.0f && s.dy[k] == 0.0f && s.dz[k] == 0.0f && s.w[k] == 0.0f && s.dw[k] == 0.0f;
  return __all_sync(0xFFFFFFFFu, ok) && isvalidf(s.numSamples) && s.numSamples >= 0.0f && isvalidf(s.sumWeights) &&
         s.sumWeights >= 0.0f;
}
__device__ void split_clear(SplitState &s, uint32_t K) {
  s.K = K;
  int c = vec_count(int(K));
  for (int k = 0; k < c * kLanes; ++k)
    s.chi2[k] = s.cx[k] = s.cy[k] = s.cz[k] = s.mx[k] = s.my[k] = s.n[k] = s.sw[k] = s.sa[k] = 0.0f;
}
__device__ void split_zero_lane(SplitState &s, int i) {
  s.chi2[i] = s.sa[i] = s.n[i] = s.sw[i] = s.mx[i] = s.my[i] = s.cx[i] = s.cy[i] = s.cz[i] = 0.0f;
}
__device__ void split_decay(SplitState &s, float a) {
  int c = vec_count(int(s.K));
  for (int k = 0; k < c * kLanes; ++k) { s.cx[k] *= a; s.cy[k] *= a; s.cz[k] *= a; s.n[k] *= a; s.sw[k] *= a; s.sa[k] *= a; }
}
__device__ bool split_is_valid(const SplitState &s) {
  const int k = threadIdx.x & 31;
  const bool ok = isvalidf(s.mx[k]) && isvalidf(s.my[k]) && isvalidf(s.cx[k]) && isvalidf(s.cy[k]) &&
                  isvalidf(s.cz[k]) && isvalidf(s.chi2[k]) && s.chi2[k] >= 0.0f && isvalidf(s.sw[k]) &&
                  s.sw[k] >= 0.0f && isvalidf(s.sa[k]) && s.sa[k] >= 0.0f && isvalidf(s.n[k]) && s.n[k] >= 0.0f;
  // a vector lane is good when it is in all four lobe vectors; one good lane is enough
  const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
  return (m & m >> 8 & m >> 16 & m >> 24 & 0xFFu) != 0 && s.K > 0 && s.K <= kMaxK;
}

// The statistics' normalisation (WEMFactory.h:553-572) and the MAP M-step
// (WEMFactory.h:895-1148; mask == nullptr is the full step) by one warp, lane k
// doing lobe k; the sums over lobes keep the reference's order (vfloat8 lane sums
// over k, then the 8-lane reduction) on lane 0.
__device__ void suff_normalize_warp(SuffState &s, float n) {
  const unsigned full = 0xFFFFFFFFu;
  const int k = int(threadIdx.x & 31);
  const int Kp = vec_count(int(s.K)) * kLanes;
  float nrm = 0.0f;
  if (k == 0) {
    s.numSamples = n;
    float sv[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = 0; j < Kp; ++j) sv[j % kLanes] += s.w[j];
    s.sumWeights = reduce8(sv);
    nrm = n / s.sumWeights;
    s.normalized = 1;
  }
  nrm = __shfl_sync(full, nrm, 0);  // lane 0 has read every weight
  if (k < Kp) {
    s.dx[k] *= nrm;
    s.dy[k] *= nrm;
    s.dz[k] *= nrm;
    s.w[k] *= nrm;
  }
  __syncwarp();
}
__device__ void map_step_warp(VMMState &v, const SuffState &cur, const SuffState &prev, const FieldConfig &cfg,
                              const int *mask) {
  const unsigned full = 0xFFFFFFFFu;
  const int k = int(threadIdx.x & 31);
  const int c = vec_count(int(v.K)), Kp = c * kLanes;
  const bool act = k < Kp;
  const float K = float(v.K);
  const float N = cur.numSamples + prev.numSamples;
  const int rem = int(v.K % kLanes);
  if (!mask) {
    if (act) {
      const float w = cur.w[k] + prev.w[k];
      v.w[k] = (cfg.weightPrior + w) / ((cfg.weightPrior * K) + N);
    }
  } else {
    float wNew = 0.0f, wOld = 0.0f;
    int m = 0;
    if (act) {
      const float w = cur.w[k] + prev.w[k];
      wNew = (cfg.weightPrior + w) / ((cfg.weightPrior * K) + N);
      wOld = v.w[k];
      m = mask[k];
    }
    // lane sums over the lobes in order, on lane 0
    float sw[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0}, sp[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = 0; j < Kp; ++j) {
      const float pj = __shfl_sync(full, m ? wNew : 0.0f, j);
      const float wj = __shfl_sync(full, m ? 0.0f : wOld, j);
      sp[j % kLanes] += pj;
      sw[j % kLanes] += wj;
    }
    float inv = 0.0f;
    if (k == 0) {
      inv = 1.0f / reduce8(sp);
      inv *= 1.0f - reduce8(sw);
    }
    inv = __shfl_sync(full, inv, 0);
    if (act) v.w[k] = m ? wNew * inv : wOld;
  }
  if (rem > 0 && k >= (c - 1) * kLanes + rem && k < Kp) v.w[k] = 0.0f;

  const float curN = cur.numSamples, prevN = prev.numSamples, NN = curN + prevN;
  const float overallN = cur.numSamples + prev.overallNumSamples;
  const float curW = curN / NN, prevW = 1.0f - curW;
  if (act) {
    const float partialN = v.w[k] * overallN;
    const V3 cm = cur.w[k] > 0.0f ? mk(cur.dx[k] / cur.w[k], cur.dy[k] / cur.w[k], cur.dz[k] / cur.w[k]) : mk(0, 0, 0);
    const V3 pm =
        prev.w[k] > 0.0f ? mk(prev.dx[k] / prev.w[k], prev.dy[k] / prev.w[k], prev.dz[k] / prev.w[k]) : mk(0, 0, 0);
    const V3 md = cm * curW + pm * prevW;
    float mc = length(md);
    const bool upd = mask ? (mask[k] != 0) : true;
    if (upd && mc > 0.0f) {
      v.mx[k] = md.x / mc;
      v.my[k] = md.y / mc;
      v.mz[k] = md.z / mc;
    }
    mc = (cfg.mcPrior * cfg.mcPriorStrength + mc * partialN) / (cfg.mcPriorStrength + partialN);
    mc = emin(cfg.maxMeanCosine, mc);
    if (upd) {
      v.mc[k] = mc;
      v.kappa[k] = mean_cosine_to_kappa(mc);
    }
    if (rem > 0 && k >= (c - 1) * kLanes + rem) {
      v.mx[k] = 0.0f; v.my[k] = 0.0f; v.mz[k] = 1.0f; v.mc[k] = 0.0f; v.kappa[k] = 0.0f;
      if (!mask) { v.norm[k] = kInv4Pi; v.e2k[k] = 1.0f; }
    }
    // vmm_calc_norm for lobe k
    v.e2k[k] = fexp(-2.0f * v.kappa[k]);
    const float nrm = v.kappa[k] / (kTwoPiF * (1.0f - v.e2k[k]));
    v.norm[k] = v.kappa[k] > 0.0f ? nrm : kInv4Pi;
  }
  __syncwarp();
}

__device__ void map3d_to_2d(V3 d, float &x, float &y) {  // Splitter.h:161-171
  float alpha = facos(d.z);
  float inv_sinc = alpha / fsin(alpha);
  x = alpha > 0.0f ? d.x * inv_sinc : 0.0f;
  y = alpha > 0.0f ? d.y * inv_sinc : 0.0f;
}
__device__ V3 map2d_to_3d(float x, float y) {  // Splitter.h:174-186
  float len = sqrtf(x * x + y * y);
  float sinc = fsin(len) / len;
  V3 r;
  r.x = len > 0.0f ? x * sinc : 0.0f;
  r.y = len > 0.0f ? y * sinc : 0.0f;
  r.z = lib_cosf(len);
  return r;
}

// SplitComponent (Splitter.h:527-665): what becomes of component idx, false
// when it is not split.
struct SplitLobes {
  float w;  // of either
  V3 m0, m1;
  float mc0, mc1;
};
__device__ bool split_component(const VMMState &v, const SplitState &sp, int idx, const FieldConfig &cfg, SplitLobes &o) {
  float numAssigned = sp.sa[idx];
  float invSW = rcp_avx2(sp.sw[idx]);
  float meanx = sp.mx[idx], meany = sp.my[idx];
  float cx = sp.cx[idx] * invSW, cy = sp.cy[idx] * invSW, cz = sp.cz[idx] * invSW;
  float D = sqrtf((cx - cy) * (cx - cy) + ((cz * cz) * 4.0f)) * 0.5f;
  float ev0 = float(double(cx + cy) * 0.5);
  ev0 += D;
  float e0x = -cz, e0y = cx - ev0;
  float l0 = sqrtf(e0x * e0x + e0y * e0y);
  e0x /= l0;
  e0y /= l0;
  float w = v.w[idx], mc = v.mc[idx], kappa = v.kappa[idx];
  if (double(kappa) >= double(cfg.maxKappaSplit) * 0.9) return false;
  V3 mu = mk(v.mx[idx], v.my[idx], v.mz[idx]);
  o.w = w * 0.5f;
  o.m0 = o.m1 = mu;
  o.mc0 = mc;
  o.mc1 = mc * mc;
  if (D > 1e-8f) {
    float ax = (e0x * ev0) * 0.5f, ay = (e0y * ev0) * 0.5f;
    Frame fr = frame_of(mu, false);
    o.m0 = xfm(fr, map2d_to_3d(meanx + ax, meany + ay));
    o.mc0 = mc / fabsf(dot(mu, o.m0));
    o.mc0 = smin(o.mc0, cfg.maxMeanCosineSplit);
    o.mc1 = o.mc0;
    o.m1 = xfm(fr, map2d_to_3d(meanx - ax, meany - ay));
  } else {
    if (numAssigned < 2.0f) return false;
  }
  return true;
}

// ---------------------------------------------------------------- merge cost (parallel over pairs)
__device__ float product_scale(V3 m0, float k0, float n0, V3 m1, float k1, float n1, V3 &pm, float &pk, float &pn) {
  pm = m0 * k0 + m1 * k1;  // Merger.h:368-396
  pk = sqrtf(dot(pm, pm));
  pn = float(1.0 / (4.0 * kPiD));
  if (pk > 1e-3f) {
    float pe = lib_expf(-2.0f * pk);
    pn = vmf_norm_double(pk, pe);
    pm = pm / pk;
  } else {
    pk = 0.0f;
    pm = m0;
  }
  float scale = (n0 * n1) / pn;
  float c0 = dot(m0, pm), c1 = dot(m1, pm);
  scale *= lib_expf(k0 * (c0 - 1.0f) + k1 * (c1 - 1.0f));
  return scale;
}
__device__ float integrated_division(V3 m0, float k0, float n0, V3 m1, float k1, float n1, float e2k1) {  // Merger.h:337-365
  V3 pm = m0 * k0 + m1 * k1;
  float pk = sqrtf(dot(pm, pm));
  float pn = float(1.0 / (4.0 * kPiD));
  if (pk > 1e-3f) {
    float pe = lib_expf(-2.0f * pk);
    pn = vmf_norm_double(pk, pe);
    pm = pm / pk;
  } else {
    pm = m0;
  }
  float scale = (n0 * n1) / pn;
  float c0 = dot(m0, pm), c1 = dot(m1, pm);
  scale = scale_norm_double(scale, e2k1, k1 * k1);
  scale *= lib_expf((k0 * (c0 - 1.0f) + k1 * (c1 - 1.0f)) + (2.0f * k1));
  return scale;
}
// The merged lobe of components i0 and i1 (Merger.h:92-133).
__device__ void merged_lobe(const VMMState &v, int i0, int i1, V3 &m, float &kappa, float &nrm, float &e2k) {
  const float w0 = v.w[i0], mc0 = v.mc[i0], w1 = v.w[i1], mc1 = v.mc[i1];
  const V3 m0 = mk(v.mx[i0], v.my[i0], v.mz[i0]), m1 = mk(v.mx[i1], v.my[i1], v.mz[i1]);
  const float w = w0 + w1;
  kappa = 0.0f;
  nrm = kInv4Pi;
  e2k = 1.0f;
  m = m0 * (w0 * mc0) + m1 * (w1 * mc1);
  m = m / w;
  float mc = m.x * m.x + m.y * m.y + m.z * m.z;
  if (mc > 0.f) {
    mc = sqrtf(mc);
    kappa = mean_cosine_to_kappa(mc);
    kappa = kappa < 1e-3f ? 0.f : kappa;
    e2k = lib_expf(-2.0f * kappa);
    nrm = vmf_norm_double(kappa, e2k);
    m = m / mc;
  } else {
    m = m0;
  }
}
// Merge costs (Merger.h:92-177) of the first nP pairs of M.i, M.j (255: none)
// into S.cost, by the whole block.  A cost is the merged lobe, the products of
// the two components with themselves and with each other, and the integral of
// each product over the merged lobe; computed by one thread it was one chain of
// 20,000 cycles, twenty times per region.  Here a thread takes one part of one
// cost: merged lobes and products first (warps of either), then the three
// integrals of each pair, then their sum.  A component's product with itself
// serves all its pairs: it is made anew for the components with `selves` set.
__device__ void merge_costs(EmShared &S, int nP, uint32_t selves) {
  MergeParts &M = S.merge;
  const VMMState &v = S.vmm;
  const int nPad = (nP + 31) & ~31;
  for (int x = threadIdx.x; x < 2 * nPad + kMaxK; x += kEmThreads) {
    if (x < nPad) {
      if (x >= nP || M.i[x] == 255) continue;
      V3 m;
      merged_lobe(v, M.i[x], M.j[x], m, M.kappa[x], M.norm[x], M.e2k[x]);
      M.mx[x] = m.x;
      M.my[x] = m.y;
      M.mz[x] = m.z;
      continue;
    }
    const bool self = x >= 2 * nPad;
    const int q = x - nPad, c = x - 2 * nPad;
    if (self ? !(selves >> c & 1u) : q >= nP || M.i[q] == 255) continue;
    const int i = self ? c : M.i[q], j = self ? c : M.j[q];
    V3 pm;
    float pk, pn;
    const float scale = product_scale(mk(v.mx[i], v.my[i], v.mz[i]), v.kappa[i], v.norm[i],
                                      mk(v.mx[j], v.my[j], v.mz[j]), v.kappa[j], v.norm[j], pm, pk, pn);
    const int o = self ? kMergePairs + c : q;
    M.px[o] = pm.x;
    M.py[o] = pm.y;
    M.pz[o] = pm.z;
    M.pkappa[o] = pk;
    M.pnorm[o] = pn;
    M.pscale[o] = scale;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < 3 * nPad; x += kEmThreads) {
    const int t = x / nPad, q = x - t * nPad;
    if (q >= nP || M.i[q] == 255) continue;
    const int o = t == 0 ? kMergePairs + M.i[q] : (t == 1 ? kMergePairs + M.j[q] : q);
    M.part[t][q] = M.pscale[o] * integrated_division(mk(M.px[o], M.py[o], M.pz[o]), M.pkappa[o], M.pnorm[o],
                                                     mk(-M.mx[q], -M.my[q], -M.mz[q]), M.kappa[q], M.norm[q], M.e2k[q]);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nP; q += kEmThreads) {
    const int i = M.i[q], j = M.j[q];
    if (i == 255) continue;
    const float w0 = v.w[i], w1 = v.w[j], w = w0 + w1;
    const float w00 = w0 * w0, w11 = w1 * w1, w01 = w0 * w1;
    float chi = 0.0f;
    chi += (w00 / w) * M.part[0][q];
    chi += (w11 / w) * M.part[1][q];
    chi += 2.0f * (w01 / w) * M.part[2][q];
    chi -= w;
    S.cost[i][j] = chi;
  }
}
// ComponentSplitStatistics::mergeComponentStats, zero-mean form (Splitter.h:994-1100)
__device__ void split_merge_stats(SplitState &s, int I, int J, float wI, V3 muI, float wJ, V3 muJ, float wK, V3 muK) {
  int L = int(s.K) - 1;
  Frame invK = inverse_of(frame_of(muK, false));
  float ix, iy, jx, jy;
  map3d_to_2d(xfm(invK, muI), ix, iy);
  map3d_to_2d(xfm(invK, muJ), jx, jy);
  float invWK = (wK > 0.f) ? rcp_avx2(wK) : 1.f;
  float swI = s.sw[I], swJ = s.sw[J], swK = swI + swJ;
  V3 cI = (swI > 0.f) ? mk(s.cx[I], s.cy[I], s.cz[I]) * rcp_avx2(swI) : mk(0, 0, 0);
  V3 cJ = (swJ > 0.f) ? mk(s.cx[J], s.cy[J], s.cz[J]) * rcp_avx2(swJ) : mk(0, 0, 0);
  V3 mII = mk(ix * ix, iy * iy, ix * iy), mJJ = mk(jx * jx, jy * jy, jx * jy);
  V3 cK = ((cI * wI + mII * wI) + cJ * wJ) + mJJ * wJ;
  cK = cK * invWK;
  V3 scK = cK * swK;
  float saK = s.sa[I] + s.sa[J];
  float nK = invWK * (wI * s.n[I] + wJ * s.n[J]);
  float chiK = s.chi2[I] + s.chi2[J];
  s.mx[I] = 0.0f; s.my[I] = 0.0f; s.cx[I] = scK.x; s.cy[I] = scK.y; s.cz[I] = scK.z;
  s.sw[I] = swK; s.n[I] = nK; s.sa[I] = saK; s.chi2[I] = chiK;
  s.mx[J] = s.mx[L]; s.my[J] = s.my[L]; s.cx[J] = s.cx[L]; s.cy[J] = s.cy[L]; s.cz[J] = s.cz[L];
  s.sw[J] = s.sw[L]; s.n[J] = s.n[L]; s.sa[J] = s.sa[L]; s.chi2[J] = s.chi2[L];
  split_zero_lane(s, L);
  s.K--;
}

// ---------------------------------------------------------------- sample passes
//
// Distance and split-statistics passes run in the home block as a two-stage
// pipeline over chunks of samples, with one __syncthreads per chunk and two
// shared-memory stages: producer warps write a chunk's terms to stage (c & 1)
// while consumer lanes add the chunk in stage ((c - 1) & 1) in sample order,
// a lane per lobe.  The consumers keep the reference's summation order
// (sequential over samples within each SIMD lane).  Samples that the reference
// skips (pdf <= 1e-16) contribute a term of exactly +-0, which leaves an
// accumulator unchanged: accumulators start at +0 and a round-to-nearest sum
// that starts at +0 never becomes -0.  E-step passes (most of the work) use the
// same roles, with a loader warp besides, and can take chunks made by other
// blocks (below).

struct LeafSamples {
  const float4 *dirw;  // direction xyz, weight
  const float *pdf;
  const float *dist;
  uint32_t count;
};

// x86 RCPSS from the block's shared copy of the table (per-lane gathers from
// constant memory would serialise)
__device__ __forceinline__ float rcp_avx2_tab(float a, const uint32_t *tab) {
  uint32_t u = f2u(a), s = u & 0x80000000u, e = (u >> 23) & 0xFFu, m = u & 0x7FFFFFu;
  float r;
  if (e == 0) {
    r = u2f(s | 0x7F800000u);
  } else if (e == 255) {
    r = m ? a : u2f(s);
  } else {
    uint32_t t = tab[m >> 12];
    int re = int((t >> 23) & 0xFFu) - (int(e) - 127);
    r = re <= 0 ? u2f(s) : (re >= 255 ? u2f(s | 0x7F800000u) : u2f(s | (uint32_t(re) << 23) | (t & 0x7FFFFFu)));
  }
  return r * fmaf_(-r, a, 2.0f);
}

// The lobe parameters of a pass by pairs of lobes, for packed arithmetic:
// {x0, x1, y0, y1}, {z0, z1, kappa0, kappa1}, {norm0, norm1, w0, w1}.
__device__ void pack_pairs(EmShared &S, int Kp) {
  const int k = 2 * int(threadIdx.x);
  if (k < Kp) {
    const VMMState &v = S.vmm;
    float4 *o = S.lobeP + pair_at(k);
    o[0] = make_float4(v.mx[k], v.mx[k + 1], v.my[k], v.my[k + 1]);
    o[1] = make_float4(v.mz[k], v.mz[k + 1], v.kappa[k], v.kappa[k + 1]);
    o[2] = make_float4(v.norm[k], v.norm[k + 1], v.w[k], v.w[k + 1]);
  }
}

// Two lobes' terms w norm fexp(kappa min(cos - 1, 0)) of direction d, the
// multiplications packed.  The exponential's argument is not positive (or
// NaN): below -100 the result is 0 either way, so the argument is clamped there
// (NaN kept) and the scale's exponent clamped at 0; the rest is fexp's.
__device__ __forceinline__ float2 pair_terms(const float4 *P, V3 d) {
  const float ln2Part1 = float(0.6931457519), ln2Part2 = float(1.4286067653e-6);
  const float4 xy = P[0], zk = P[1], nw = P[2];
  float2 c = mul2(f2(d.z), make_float2(zk.x, zk.y));
  c = fma2(f2(d.y), make_float2(xy.z, xy.w), c);
  c = fma2(f2(d.x), make_float2(xy.x, xy.y), c);
  // fminf(NaN, 0) is 0, as the reference's MINPS
  float2 v = mul2(make_float2(zk.z, zk.w), make_float2(fminf(c.x - 1.0f, 0.0f), fminf(c.y - 1.0f, 0.0f)));
  asm("max.NaN.f32 %0, %0, 0fC2C80000;" : "+f"(v.x));  // -100
  asm("max.NaN.f32 %0, %0, 0fC2C80000;" : "+f"(v.y));
  const float2 sc = mul2(v, f2(1.44269502162933349609375f));
  const float t0 = __fadd_rd(sc.x, 12582912.0f), t1 = __fadd_rd(sc.y, 12582912.0f);  // floor, see fexp
  const float2 kr = make_float2(t0 - 12582912.0f, t1 - 12582912.0f);
  const uint32_t e0 = uint32_t(max(int(f2u(t0)) - (0x4B400000 - 127), 0)) << 23;
  const uint32_t e1 = uint32_t(max(int(f2u(t1)) - (0x4B400000 - 127), 0)) << 23;
  float2 m = mul2(kr, f2(ln2Part1));
  float2 x = make_float2(v.x - m.x, v.y - m.y);
  m = mul2(kr, f2(ln2Part2));
  x = make_float2(x.x - m.x, x.y - m.y);
  float2 r = mul2(x, f2(2.7555381529964506626129150390625e-4f));
  const float coeff[7] = {1.304379315115511417388916015625e-3f, 8.378830738365650177001953125e-3f,
                          4.16539050638675689697265625e-2f, 0.166668415069580078125f,
                          0.4999999105930328369140625f, 1.0f, 1.0f};
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    r = make_float2(r.x + coeff[i], r.y + coeff[i]);
    r = i < 6 ? mul2(x, r) : mul2(r, make_float2(u2f(e0), u2f(e1)));
  }
  return mul2(make_float2(nw.z, nw.w), mul2(make_float2(nw.x, nw.y), r));
}

// a / b in a function of its own: as a plain expression behind a condition the
// compiler evaluates the division for every operand and selects afterwards,
// and most lobes are far from a sample's direction, so that most numerators
// would run its slow path for small operands.
__device__ __noinline__ float div_plain(float a, float b) { return a / b; }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}

// ---- distance passes (WEMFactory.h:1199-1326): per lobe the sums of wts and of
// wts * rcp(distance), wts = (w a) (a pdf / weight).  A sample per producer
// thread as in the E-step (below); a chunk holds rows wts_k (0 for skipped
// samples) and rcp(distance) of RS = C + 4 floats; one consumer warp, lane k
// summing both chains of lobe k.  22 cycles per sample at 23 lobes, issue bound in
// the producers; 50 with a lane per lobe vector and two rows per lobe.
template <int kCnt>
__device__ __noinline__ void produce_distance(const EmShared &S, int RS, float4 dw, float dist, bool have, float *row) {
  constexpr int Kp = kCnt * kLanes;
  const V3 d = mk(dw.x, dw.y, dw.z);
  const float w = dw.w;
  float2 term[Kp / 2], p[kLanes / 2];
#pragma unroll
  for (int v = 0; v < kCnt; ++v)
#pragma unroll
    for (int j = 0; j < kLanes / 2; ++j) {
      const int i = v * (kLanes / 2) + j;
      term[i] = pair_terms(S.lobeP + pair_at(2 * i), d);
      p[j] = v == 0 ? term[i] : make_float2(p[j].x + term[i].x, p[j].y + term[i].y);
    }
  const float pdf = ((p[0].x + p[0].y) + (p[1].x + p[1].y)) + ((p[2].x + p[2].y) + (p[3].x + p[3].y));  // reduce8
  const bool valid = have && pdf > 1e-16f;
  const float inv = valid ? rcp_avx2_tab(pdf, S.rcpTab) : 0.0f;
  row[Kp * RS] = valid ? rcp_avx2_tab(dist, S.rcpTab) : 0.0f;
  bool redo = false;
#pragma unroll
  for (int i = 0; i < Kp / 2; ++i) {
    const float2 wy0 = S.lobeW[2 * i], wy1 = S.lobeW[2 * i + 1];
    const float2 a = mul2(term[i], f2(inv));
    const float2 n = mul2(a, f2(pdf));
    const bool s0 = n.x < kSmallNumerator, s1 = n.y < kSmallNumerator;
    const float2 q = pair_quotients(n, make_float2(wy0.x, wy1.x), make_float2(wy0.y, wy1.y),
                                    make_float2(s0 ? 0x1p50f : 1.0f, s1 ? 0x1p50f : 1.0f),
                                    make_float2(s0 ? 0x1p-50f : 1.0f, s1 ? 0x1p-50f : 1.0f));
    const float2 wts = mul2(mul2(f2(w), a), q);
    row[2 * i * RS] = valid ? wts.x : 0.0f;
    row[(2 * i + 1) * RS] = valid ? wts.y : 0.0f;
    // a numerator out of range, a weight out of [1e-8, 1e8] (marked by a zero reciprocal)
    redo |= !(n.x <= 1e15f) | !(n.y <= 1e15f) | (wy0.y == 0.0f) | (wy1.y == 0.0f);
  }
  if (redo && valid) {
#pragma unroll 1
    for (int k = 0; k < Kp; ++k) {
      const float a = __fmul_rn((k & 1) ? pair_terms(S.lobeP + pair_at(k), d).y : pair_terms(S.lobeP + pair_at(k), d).x, inv);
      row[k * RS] = (w * a) * div_plain(a * pdf, S.lobeW[k].x);
    }
  }
}

template <int kCnt>
__device__ __noinline__ void run_distance(EmShared &S, const LeafSamples &L) {
  constexpr int Kp = kCnt * kLanes;
  constexpr int P = kEmThreads - 32;  // one consumer warp
  constexpr int C = P, RS = C + 4;
  static_assert((Kp + 1) * RS <= kStageFloats, "a distance chunk fits its stage");
  const int tid = threadIdx.x;
  const uint32_t rounds = (L.count + C - 1) / C;
  const bool producer = tid < P;
  float4 dw = make_float4(0.f, 0.f, 0.f, 0.f);
  float dist = 0.0f;
  if (producer && uint32_t(tid) < L.count) {
    dw = L.dirw[tid];
    dist = L.dist[tid];
  }
  const int k = min(tid & 31, Kp - 1);
  float sumD = 0.0f, sumW = 0.0f;
  for (uint32_t it = 0; it <= rounds; ++it) {
    if (producer && it < rounds) {
      const uint32_t idx = it * C + uint32_t(tid), nextIdx = idx + C;
      const float4 cur = dw;
      const float curDist = dist;
      if (nextIdx < L.count) {
        dw = L.dirw[nextIdx];
        dist = L.dist[nextIdx];
      }
      produce_distance<kCnt>(S, RS, cur, curDist, idx < L.count, S.pbuf + (it & 1) * kStageFloats + tid);
    }
    if (!producer && it >= 1) {
      const uint32_t base = smem_u32(S.pbuf + ((it - 1) & 1) * kStageFloats);
      uint32_t A = base + uint32_t(k * RS) * 4u, D = base + uint32_t(Kp * RS) * 4u;
      const int n = int(min(uint32_t(C), L.count - (it - 1) * C));
      const int n8 = (n + 7) & ~7;
      float4 a0 = lds4(A), d0 = lds4(D), a1 = lds4(A + 16), d1 = lds4(D + 16);
#pragma unroll 1
      for (int s = 0; s < n8; s += 8) {
        A += 32;
        D += 32;
        const float2 p0 = mul2(make_float2(a0.x, a0.y), make_float2(d0.x, d0.y));
        const float2 p1 = mul2(make_float2(a0.z, a0.w), make_float2(d0.z, d0.w));
        const float2 p2 = mul2(make_float2(a1.x, a1.y), make_float2(d1.x, d1.y));
        const float2 p3 = mul2(make_float2(a1.z, a1.w), make_float2(d1.z, d1.w));
        const float4 v0 = a0, v1 = a1;
        a0 = lds4(A);  // the last turn's loads run up to 8 floats past the row
        d0 = lds4(D);
        a1 = lds4(A + 16);
        d1 = lds4(D + 16);
        sumD += p0.x; sumW += v0.x;
        sumD += p0.y; sumW += v0.y;
        sumD += p1.x; sumW += v0.z;
        sumD += p1.y; sumW += v0.w;
        sumD += p2.x; sumW += v1.x;
        sumD += p2.y; sumW += v1.y;
        sumD += p3.x; sumW += v1.z;
        sumD += p3.y; sumW += v1.w;
      }
    }
    __syncthreads();
  }
  if (!producer && (tid & 31) < Kp) {
    S.xch[0][k] = sumD;
    S.xch[1][k] = sumW;
  }
  __syncthreads();
}

// ---- split-statistics passes (Splitter.h:439-523).  Producers: kCnt adjacent
// lanes per sample, one lobe vector each (the vectors' pdf sums carried from
// lane to lane in order); a chunk holds, per lobe, rows a, x and y of the
// direction in the lobe's frame, and chi (all 0 for skipped samples), then
// the rows of the sample's weight and validity.  Rows hold RS floats (a
// multiple of four, RS / 4 odd) and the parts' blocks of rows start a few banks
// apart, so that the parts of a sample store to distinct banks.  Consumers: warp 14, lane k
// summing lobe k's a, a w and (a w)(x x), (a w)(y y), (a w)(x y); warp 15,
// lane k its running chi-square mean.  The products are formed by the
// consumers, four rows per lobe in place of seven, which makes chunks of 112 to
// 448 samples of what were 80 to 200, and the counts' reciprocals by the chi-square
// lanes.  Bound by the chi-square chain (47 cycles per sample beside the
// producers' 36 at 24 lobes; 105 while the producers made seven rows a lobe and
// counted the valid samples between two barriers).
struct SplitShape {
  int C, RS, vec, part;  // samples per chunk; floats per row, per lobe vector of rows, per part
};
template <int kCnt>
__device__ constexpr SplitShape split_shape() {
  constexpr int perWarp = 32 / kCnt;
  constexpr int C = (kEmThreads / 32 - 2) * perWarp;
  constexpr int RS = ((C + 4) / 8) * 8 + 4;  // > C, RS / 4 odd
  return SplitShape{C, RS, kLanes * RS, 4 * kLanes * RS + (kCnt == 2 ? 16 : kCnt == 3 ? 12 : 8)};
}

template <int kCnt>
__device__ __noinline__ void produce_split(const EmShared &S, int v, float4 dw, float spdf, bool have, float *B, int s) {
  constexpr SplitShape sh = split_shape<kCnt>();
  constexpr int RS = sh.RS;
  const unsigned full = 0xFFFFFFFFu;
  const V3 d = mk(dw.x, dw.y, dw.z);
  const float w = dw.w;
  const float4 *P = S.lobeP + v * (3 * kLanes / 2 + 1), *F = S.frameP + v * (3 * kLanes / 2 + 1);
  float2 term[kLanes / 2], p[kLanes / 2];
#pragma unroll
  for (int j = 0; j < kLanes / 2; ++j) p[j] = term[j] = pair_terms(P + 3 * j, d);
#pragma unroll
  for (int step = 1; step < kCnt; ++step)
#pragma unroll
    for (int j = 0; j < kLanes / 2; ++j) {
      const float x = __shfl_up_sync(full, p[j].x, 1), y = __shfl_up_sync(full, p[j].y, 1);
      if (v == step) p[j] = make_float2(x + term[j].x, y + term[j].y);
    }
  float pdf = ((p[0].x + p[0].y) + (p[1].x + p[1].y)) + ((p[2].x + p[2].y) + (p[3].x + p[3].y));  // reduce8
  if (kCnt > 1) pdf = __shfl_sync(full, pdf, (int(threadIdx.x) & 31) - v + kCnt - 1);  // the last part's
  const bool valid = have && pdf > 1e-16f;
  const float inv = valid ? rcp_avx2_tab(pdf, S.rcpTab) : 0.0f;
  const float value = w * spdf, vv = value * value;
  const float mc = S.mcEstimate;
  const float den1 = mc * pdf, den2 = ((mc * mc) * pdf) * pdf;
  // bounds within which nothing but a denormal quotient under- or overflows
  const bool inside = (value == 0.0f || (fabsf(value) >= 1e-4f && fabsf(value) <= 1e4f)) && den1 >= 1e-10f &&
                      den1 <= 1e4f && spdf >= 1e-6f && spdf <= 1e6f;
  const float y1 = rcp_newton(den1), y2 = rcp_newton(den2), y3 = rcp_newton(spdf);
  bool redo = !inside;
  float *row = B + v * sh.part + s;
#pragma unroll
  for (int j = 0; j < kLanes / 2; ++j) {
    const float2 a = mul2(term[j], f2(inv));
    const float2 vmf = mul2(a, f2(pdf));
    const bool s0 = vmf.x < kSmallNumerator, s1 = vmf.y < kSmallNumerator;
    const float2 up = make_float2(s0 ? 0x1p50f : 1.0f, s1 ? 0x1p50f : 1.0f);
    const float2 down = make_float2(s0 ? 0x1p-50f : 1.0f, s1 ? 0x1p-50f : 1.0f);
    const float2 pvp = pair_quotients(mul2(vmf, f2(value)), f2(den1), f2(y1), up, down);
    float2 chi = pair_quotients(mul2(f2(vv), vmf), f2(den2), f2(y2), up, down);
    const float2 two = mul2(f2(2.0f), pvp);
    chi = make_float2((chi.x - two.x) + vmf.x, (chi.y - two.y) + vmf.y);
    chi = pair_quotients(chi, f2(spdf), f2(y3), up, down);
    redo |= !(fabsf(chi.x) <= 1e20f) | !(fabsf(chi.y) <= 1e20f);
    chi = make_float2(a.x > 0.0f ? chi.x : 0.0f, a.y > 0.0f ? chi.y : 0.0f);
    const float4 f0 = F[3 * j], f1 = F[3 * j + 1], f2v = F[3 * j + 2];
    const float2 lx = fma2(f2(d.x), make_float2(f0.x, f0.y),
                                 fma2(f2(d.y), make_float2(f0.z, f0.w), mul2(f2(d.z), make_float2(f1.x, f1.y))));
    const float2 ly =
        fma2(f2(d.x), make_float2(f1.z, f1.w),
                   fma2(f2(d.y), make_float2(f2v.x, f2v.y), mul2(f2(d.z), make_float2(f2v.z, f2v.w))));
    float *r = row + 2 * j * RS;
    r[0] = valid ? a.x : 0.0f;
    r[RS] = valid ? a.y : 0.0f;
    r += sh.vec;
    r[0] = valid ? lx.x : 0.0f;
    r[RS] = valid ? lx.y : 0.0f;
    r += sh.vec;
    r[0] = valid ? ly.x : 0.0f;
    r[RS] = valid ? ly.y : 0.0f;
    r += sh.vec;
    r[0] = valid ? chi.x : 0.0f;
    r[RS] = valid ? chi.y : 0.0f;
  }
  if (v == 0) {
    float *r = B + kCnt * sh.part + s;
    r[0] = valid ? w : 0.0f;
    r[RS] = valid ? 1.0f : 0.0f;
  }
  if (redo && valid) {
#pragma unroll 1
    for (int j = 0; j < kLanes; ++j) {
      const float2 t = pair_terms(P + 3 * (j / 2), d);
      const float a = __fmul_rn((j & 1) ? t.y : t.x, inv);
      const float vmf = a * pdf;
      const float pvp = div_plain(vmf * value, den1);
      float chi = div_plain(vv * vmf, den2);
      chi -= 2.0f * pvp;
      chi += vmf;
      chi = div_plain(chi, spdf);
      row[3 * sh.vec + j * RS] = a > 0.0f ? chi : 0.0f;
    }
  }
}

// Warp 14: five chains per lane over one chunk; A: the lobe's first row
// (bytes), V: bytes from its a row to its x row and from x to y, W: the weights.
struct SplitSums {
  float sa, sw, cx, cy, cz;
};
__device__ __forceinline__ void split_sums(uint32_t A, uint32_t V, uint32_t W, int n4, SplitSums &q) {
  uint32_t X = A + V, Y = X + V;
  float4 a = lds4(A), x = lds4(X), y = lds4(Y), w = lds4(W);
#pragma unroll 1
  for (int s = 0; s < n4; s += 4) {
    A += 16;
    X += 16;
    Y += 16;
    W += 16;
    const float4 a1 = lds4(A), x1 = lds4(X), y1 = lds4(Y), w1 = lds4(W);  // the last turn's run past the rows
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 ah = h ? make_float2(a.z, a.w) : make_float2(a.x, a.y);
      const float2 xh = h ? make_float2(x.z, x.w) : make_float2(x.x, x.y);
      const float2 yh = h ? make_float2(y.z, y.w) : make_float2(y.x, y.y);
      const float2 wh = h ? make_float2(w.z, w.w) : make_float2(w.x, w.y);
      const float2 aw = mul2(ah, wh);
      const float2 xx = mul2(aw, mul2(xh, xh));
      const float2 yy = mul2(aw, mul2(yh, yh));
      const float2 xy = mul2(aw, mul2(xh, yh));
      q.sa += ah.x;
      q.sw += aw.x;
      q.cx += xx.x;
      q.cy += yy.x;
      q.cz += xy.x;
      q.sa += ah.y;
      q.sw += aw.y;
      q.cx += xx.y;
      q.cy += yy.y;
      q.cz += xy.y;
    }
    a = a1;
    x = x1;
    y = y1;
    w = w1;
  }
}

// Warp 15: the running mean chi2 += (chi - chi2) / n over the valid samples of a
// chunk, n the lane's running count.  Markstein's steps with y = RN(1 / n)
// (one Newton step, a group of four samples ahead of the additions) give
// (chi - chi2) / n exactly (a skipped sample, y = 0, adds +-0) when the
// difference d and the quotient lie in [1e-30, 1e30] (or d is 0).  The chain
// is five dependent operations per sample, about 21 cycles; what runs beside
// it is kept small (31 cycles per sample alone, 47 with the range checks per
// group and a guarded n): a mean stays between its start and its samples, so
// their sizes bound d, and the smallest non-zero |d| of the chunk is held against
// 1e-30 times its last n, so every quotient is in range.  A chunk that fails
// (rare) is summed again with divisions, which give the same bits wherever
// Markstein's steps were exact.  kGuard: a count may be 0 before the first valid
// sample.
template <bool kGuard>
__device__ __forceinline__ void chi_counts(float n0, float4 v, float4 &n, float4 &r) {
  n.x = n0 + v.x;
  n.y = n.x + v.y;
  n.z = n.y + v.z;
  n.w = n.z + v.w;
  r.x = rcp_newton(kGuard ? fmaxf(n.x, 0.5f) : n.x) * v.x;  // n >= 1 where v is not 0
  r.y = rcp_newton(kGuard ? fmaxf(n.y, 0.5f) : n.y) * v.y;
  r.z = rcp_newton(kGuard ? fmaxf(n.z, 0.5f) : n.z) * v.z;
  r.w = rcp_newton(kGuard ? fmaxf(n.w, 0.5f) : n.w) * v.w;
}
template <bool kGuard>
__device__ __forceinline__ void split_chi(const float *xr, const float *vr, int n4, float &acc, float &accN) {
  const float accStart = acc, nStart = accN;
  uint32_t X = smem_u32(xr), V = smem_u32(vr);
  float hi = fabsf(acc);       // largest |chi|, and the mean at the start
  uint32_t lo = 0xFFFFFFFFu;  // smallest non-zero |d|, as twice its bits minus one (a zero's are the largest)
  float4 x = lds4(X), v = lds4(V), n, r;
  chi_counts<kGuard>(accN, v, n, r);
  v = lds4(V + 16);
#pragma unroll 2
  for (int s = 0; s < n4; s += 4) {
    X += 16;
    V += 16;
    const float4 x1 = lds4(X), v1 = lds4(V + 16);  // the last turns' loads run past the rows
    float4 nn, rn;
    chi_counts<kGuard>(n.w, v, nn, rn);
    const float d1 = x.x - acc;
    acc = acc + markstein_q(d1, n.x, r.x);
    const float d2 = x.y - acc;
    acc = acc + markstein_q(d2, n.y, r.y);
    const float d3 = x.z - acc;
    acc = acc + markstein_q(d3, n.z, r.z);
    const float d4 = x.w - acc;
    acc = acc + markstein_q(d4, n.w, r.w);
    hi = fmaxf(fmaxf(hi, fmaxf(fabsf(x.x), fabsf(x.y))), fmaxf(fabsf(x.z), fabsf(x.w)));
    lo = min(min(lo, min(2u * f2u(d1) - 1u, 2u * f2u(d2) - 1u)), min(2u * f2u(d3) - 1u, 2u * f2u(d4) - 1u));
    accN = n.w;
    x = x1;
    v = v1;
    n = nn;
    r = rn;
  }
  if (acc != acc || !(hi <= 1e29f) || !(accN <= 1e30f) || lo < 2u * f2u(1.0000002e-30f * accN) - 1u) {
    acc = accStart;
    accN = nStart;
#pragma unroll 1
    for (int s = 0; s < n4; ++s) {
      const float vv = vr[s];
      accN += vv;
      if (vv != 0.0f) acc += div_plain(xr[s] - acc, accN);
    }
  }
}

template <int kCnt>
__device__ __noinline__ void run_split(EmShared &S, const LeafSamples &L, SplitState &sp) {
  constexpr SplitShape sh = split_shape<kCnt>();
  constexpr int Kp = kCnt * kLanes, C = sh.C, RS = sh.RS;
  constexpr int P = kEmThreads - 64;
  static_assert(kCnt * sh.part + 2 * RS <= kStageFloats, "a split chunk fits its stage");
  const int tid = threadIdx.x, lane = tid & 31;
  const uint32_t rounds = (L.count + C - 1) / C;
  const bool producer = tid < P;
  // lane l of producer warp g: part l % kCnt of the warp's sample l / kCnt (three
  // parts: lanes 30 and 31 follow along and store nothing)
  constexpr int perWarp = 32 / kCnt;
  const int v = lane % kCnt, slot = lane / kCnt;
  const bool spare = slot >= perWarp;
  const int s = (tid >> 5) * perWarp + slot;
  float4 dw = make_float4(0.f, 0.f, 0.f, 0.f);
  float spdf = 0.0f;
  if (producer && !spare && uint32_t(s) < L.count) {
    dw = L.dirw[s];
    spdf = L.pdf[s];
  }
  const int k = min(lane, Kp - 1);
  SplitSums q{};
  float chi = 0.0f, chiN = 0.0f;
  if (tid >= P && tid < P + 32) q = SplitSums{sp.sa[k], sp.sw[k], sp.cx[k], sp.cy[k], sp.cz[k]};
  if (tid >= P + 32) {
    chi = sp.chi2[k];
    chiN = sp.n[k];
  }
  long long cycP = 0, cycC = 0;
  for (uint32_t it = 0; it <= rounds; ++it) {
    const long long t0 = clock64();
    if (producer) {
      if (it < rounds) {
        const uint32_t idx = it * C + uint32_t(s), nextIdx = idx + C;
        const float4 cur = dw;
        const float curPdf = spdf;
        if (!spare && nextIdx < L.count) {
          dw = L.dirw[nextIdx];
          spdf = L.pdf[nextIdx];
        }
        // a spare lane writes to the row's padding past the chunk's last sample
        produce_split<kCnt>(S, v, cur, curPdf, !spare && idx < L.count, S.pbuf + (it & 1) * kStageFloats, spare ? RS - 1 : s);
        cycP += clock64() - t0;
      }
    } else if (it >= 1) {
      const float *B = S.pbuf + ((it - 1) & 1) * kStageFloats;
      const int n = int(min(uint32_t(C), L.count - (it - 1) * C));
      const int n4 = (n + 3) & ~3;
      const float *row = B + (k / kLanes) * sh.part + (k % kLanes) * RS, *per = B + kCnt * sh.part;
      if (tid < P + 32) split_sums(smem_u32(row), uint32_t(sh.vec) * 4u, smem_u32(per), n4, q);
      else if (__all_sync(0xFFFFFFFFu, chiN + per[RS] >= 0.5f)) split_chi<false>(row + 3 * sh.vec, per + RS, n4, chi, chiN);
      else split_chi<true>(row + 3 * sh.vec, per + RS, n4, chi, chiN);
      cycC += clock64() - t0;
    }
    __syncthreads();
  }
  if (lane < Kp) {
    if (tid >= P && tid < P + 32) {
      sp.sa[k] = q.sa;
      sp.sw[k] = q.sw;
      sp.cx[k] = q.cx;
      sp.cy[k] = q.cy;
      sp.cz[k] = q.cz;
    } else if (tid >= P + 32) {
      sp.chi2[k] = chi;
      sp.n[k] = chiN;
    }
  }
  if (tid == 0) S.prof.cycProdS += uint64_t(cycP);
  if (tid == P + 32) S.prof.cycConsS += uint64_t(cycC);
  __syncthreads();
}

// ---------------------------------------------------------------- shared E-step passes

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_acquire() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned long long *m, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *m, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *m) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *m, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return ok != 0;
}
// whether phase `parity` has completed, without waiting
__device__ __forceinline__ bool mbar_test_wait(unsigned long long *m, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return ok != 0;
}
// global -> shared bulk copy (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, unsigned long long *m) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(m))
               : "memory");
}
// orders this thread's generic-proxy global accesses with bulk copies
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void bar_named(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void set_error(int *err, int code) { atomicCAS(err, 0, code); }
__device__ __forceinline__ bool has_error(const int *err) { return *reinterpret_cast<const volatile int *>(err) != 0; }

// Spins until *p >= want (true) or the launch failed / the wait ran out
// (after limitNs; the launch's error word then holds kErrSlotWait).
__device__ bool wait_at_least(const uint32_t *p, uint32_t want, int *err, unsigned long long limitNs = kWaitNs) {
  unsigned long long t0 = 0;
  unsigned sleep = 64;
  for (uint32_t it = 0;; ++it) {
    if (ld_acquire(p) >= want) return true;
    if ((it & 31) == 31) {
      if (has_error(err)) return false;
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limitNs) {
        set_error(err, kErrSlotWait);
        return false;
      }
    }
    __nanosleep(sleep);
    sleep = sleep < 1024 ? 2 * sleep : sleep;
  }
}
// Waits for phase `parity` of a stage barrier.  Consumers give up on chunks
// from *abortAt on (the loader gave up on them: nothing will arrive); every
// waiter gives up after kWaitNs.
__device__ bool mbar_wait(unsigned long long *m, uint32_t parity, const volatile uint32_t *abortAt, uint32_t k,
                          int *err) {
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    if (mbar_try_wait(m, parity)) return true;
    if (abortAt && k >= *abortAt) return false;
    if ((it & 15) == 15) {
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitNs) {
        set_error(err, kErrCopyWait);
        return false;
      }
    }
  }
}

__device__ __forceinline__ unsigned long long grab_word(uint32_t gen, uint32_t chunks, uint32_t next) {
  return (static_cast<unsigned long long>(gen) << (2 * kGrabIdxBits)) |
         (static_cast<unsigned long long>(chunks) << kGrabIdxBits) | next;
}
__device__ __forceinline__ uint32_t grab_gen(unsigned long long w) { return uint32_t(w >> (2 * kGrabIdxBits)); }
__device__ __forceinline__ uint32_t grab_chunks(unsigned long long w) { return uint32_t(w >> kGrabIdxBits) & kGrabMask; }
__device__ __forceinline__ uint32_t grab_next(unsigned long long w) { return uint32_t(w) & kGrabMask; }
// Chunk shape of an E-step pass with `cnt` lobe vectors: a consumer warp per
// lobe vector and one for the per-sample rows (chain_role), one warp that
// loads chunks made by other blocks, the rest produce, a sample per thread,
// so that a chunk is one round of the producers.  A chunk holds rows of
// RS = C + 4 floats (RS / 4 odd, so the 128-bit loads of 8 consecutive rows
// hit distinct banks): a_k for k < Kp (the soft assignment t_k / pdf of valid
// samples, 0 otherwise), the direction x, y, z, the weight of valid samples,
// then w log(pdf) and the four unassigned-sample terms.
struct EStepShape {
  int cnt, Kp, P, cons0, consWarps, C, RS, stageFloats, stages, slots;
};
// Chunk k of a pass covers samples [chunk_begin, chunk_begin + C).
__device__ __forceinline__ uint32_t chunk_begin(const EStepShape &e, uint32_t k) { return k * uint32_t(e.C); }
__device__ __forceinline__ uint32_t chunk_count(const EStepShape &e, uint32_t count) {
  return (count + uint32_t(e.C) - 1u) / uint32_t(e.C);
}
__device__ __forceinline__ EStepShape estep_shape(int cnt, const EmTuning &tune) {
  EStepShape e;
  e.cnt = cnt;
  e.Kp = cnt * kLanes;
  e.consWarps = cnt == 4 ? 3 : cnt + 1;  // see chain_role
  e.cons0 = kEmThreads - 32 * e.consWarps;  // consumers: threads [cons0, 512)
  e.P = e.cons0 - 32;                       // producers [0, P), then the loader warp
  e.C = (min(e.P, kMaxChunk) / tune.chunkDiv) & ~15;  // chains take 16 samples at a time
  e.RS = e.C + 4;
  e.stageFloats = (e.Kp + 9) * e.RS;
  e.stages = min(min(kMaxStages, tune.stageCap), 2 * kStageFloats / e.stageFloats);
  e.slots = min(int(kRingMaxSlots), int(kRingFloats) / e.stageFloats);
  return e;
}

// Producers: `nthreads` threads (index t) fill chunk `chunk` into G (a stage
// or a ring slot), a sample per thread with the terms of all its lobes in
// registers: the lobe vectors' sums stay in order without shuffles, the 32
// lobes give independent work to cover the exponentials' latency, the lobe
// parameters are broadcast loads and a warp stores whole rows.  Issue bound:
// 30 FP32 operations and about as many issue slots per lobe, 15 cycles per
// sample at 32 lobes alone on an SM.  A lane per lobe vector and sample, with
// shuffles between the vectors, held a leaf of 30 lobes that no other block
// helps at 39 cycles per sample and pass; it now takes 28 (18 to 23 at 17 to 24
// lobes; 12 to 14 where other blocks help).
template <int kCnt>
__device__ __noinline__ void produce_estep_rows(const EmShared &S, const EStepShape &e, const float4 *dirw,
                                                uint32_t count, uint32_t chunk, float *G, int t, int nthreads) {
  constexpr int Kp = kCnt * kLanes;
  const int RS = e.RS;
  const uint32_t first = chunk_begin(e, chunk);
  for (int s = t; s < e.C; s += nthreads) {
    const uint32_t idx = first + uint32_t(s);
    const bool have = idx < count;
    const float4 dw = have ? __ldcg(dirw + idx) : make_float4(0.f, 0.f, 0.f, 0.f);
    const V3 d = mk(dw.x, dw.y, dw.z);
    float2 term[Kp / 2], p[kLanes / 2];
#pragma unroll
    for (int v = 0; v < kCnt; ++v)
#pragma unroll
      for (int j = 0; j < kLanes / 2; ++j) {
        const int i = v * (kLanes / 2) + j;
        term[i] = pair_terms(S.lobeP + pair_at(2 * i), d);
        p[j] = v == 0 ? term[i] : make_float2(p[j].x + term[i].x, p[j].y + term[i].y);
      }
    const float pdf = ((p[0].x + p[0].y) + (p[1].x + p[1].y)) + ((p[2].x + p[2].y) + (p[3].x + p[3].y));  // reduce8
    const bool valid = have && pdf > 1e-16f;
    const float inv = valid ? rcp_avx2_tab(pdf, S.rcpTab) : 0.0f;
    float *row = G + s;
#pragma unroll
    for (int i = 0; i < Kp / 2; ++i) {
      const float2 a = mul2(term[i], make_float2(inv, inv));
      row[2 * i * RS] = valid ? a.x : 0.0f;
      row[(2 * i + 1) * RS] = valid ? a.y : 0.0f;
    }
    const float w = dw.w;
    const bool un = have && !valid;
    float *X = row + Kp * RS;
    X[0] = d.x;
    X[RS] = d.y;
    X[2 * RS] = d.z;
    X[3 * RS] = valid ? w : 0.0f;
    // the log-likelihood only drives the convergence test (its relative
    // change against 0.005); it is not stored, so the single-precision
    // logf (<= 1 ulp) stands in for the C library's here
    X[4 * RS] = valid ? w * logf(pdf) : 0.0f;
    X[5 * RS] = un ? w : 0.0f;
    X[6 * RS] = un ? d.x * w : 0.0f;
    X[7 * RS] = un ? d.y * w : 0.0f;
    X[8 * RS] = un ? d.z * w : 0.0f;
  }
}
__device__ __forceinline__ void produce_estep_chunk(const EmShared &S, const EStepShape &e, const float4 *dirw,
                                                    uint32_t count, uint32_t chunk, float *G, int t, int nthreads) {
  switch (e.cnt) {
    case 1: produce_estep_rows<1>(S, e, dirw, count, chunk, G, t, nthreads); break;
    case 2: produce_estep_rows<2>(S, e, dirw, count, chunk, G, t, nthreads); break;
    case 3: produce_estep_rows<3>(S, e, dirw, count, chunk, G, t, nthreads); break;
    default: produce_estep_rows<4>(S, e, dirw, count, chunk, G, t, nthreads); break;
  }
}

// A helper takes the next chunk of board `b` (one thread): only when that
// chunk's ring slot is free (known once the pass's parameters are loaded; a
// chunk of a pass not loaded yet is taken anyway).  Returns the chunk, -1 when
// the pass has none left, -2 when the ring is full for now; `exact` says the
// chunk taken is the one whose slot was checked (others can take chunks
// between the check and the atomic).
__device__ int helper_take(EmShared &S, Board &b, bool paramsLoaded, uint32_t paramsGen, uint32_t &gen, int &exact) {
  const unsigned long long w = ld_relaxed64(&b.grab);
  const uint32_t consumed = ld_relaxed(&b.consumed);
  exact = 0;
  gen = 0;
  if (has_error(S.err) || grab_gen(w) == 0 || grab_next(w) >= grab_chunks(w)) return -1;
  const bool known = paramsLoaded && grab_gen(w) == paramsGen;
  if (known && S.hp.seqBase + grab_next(w) + 1u > consumed + uint32_t(estep_shape(int(S.hp.cnt), S.tune).slots)) return -2;
  const unsigned long long w2 = atomicAdd(&b.grab, 1ull);
  if (grab_gen(w2) == 0 || grab_next(w2) >= grab_chunks(w2)) return -1;
  gen = grab_gen(w2);
  exact = known && w2 == w;
  return int(grab_next(w2));
}

// A helper's chunk of board `b`: wait until its ring slot is free (unless
// its slot was checked), fill the slot, then publish its sequence number.
// Warp 15 holds no samples of a chunk (C <= 416), so its lane 0 takes the
// helper's next chunk meanwhile.
__device__ void produce_for(EmShared &S, Board &b, float *ring, const EStepShape &e, const float4 *dirw,
                            uint32_t count, uint32_t seqBase, uint32_t chunk, bool exact, uint32_t paramsGen) {
  const int t = threadIdx.x;
  const uint32_t seq = seqBase + chunk + 1u, slot = (seqBase + chunk) % uint32_t(e.slots);
  // the slot's previous chunk (sequence number seq - slots) must have been copied out
  if (t == 0 && !exact && seq > uint32_t(e.slots)) wait_at_least(&b.consumed, seq - uint32_t(e.slots), S.err);
  __syncthreads();
  if (t == kEmThreads - 32) {
    uint32_t g = 0;
    int x = 0;
    S.nextGrabbed = helper_take(S, b, true, paramsGen, g, x);
    S.nextGen = g;
    S.nextExact = x;
    S.hasNext = 1;
  }
  produce_estep_chunk(S, e, dirw, count, chunk, ring + size_t(slot) * e.stageFloats, t, kEmThreads);
  fence_proxy_async();  // the ring is read by bulk copies
  __syncthreads();
  if (t == 0) {
    __threadfence();
    st_release(&b.ready[slot], seq);
  }
}

// Consumer side of the sum: a_k w, (d_q a_k) w or a per-sample row, in
// sample order (the products are those of the reference's E-step).  What
// bounds a consumer warp is shared memory's way into registers: a warp's load
// returns 64 bytes per cycle whatever it shares, so a register per lane costs
// 2 cycles, and loads of 32 distinct rows of 16 bytes keep the data pipe of
// the whole SM busy for 8 (both measured on one SM).  So a warp holds the four
// chains of eight lobes, lane 8 q + j the chain q of lobe j, whose loads fetch 128
// distinct bytes: three registers per sample and chain (a, d, w), 7.3 cycles per
// sample alone, where a lane per lobe with two chains took 9.3 to 9.9.  With
// four lobe vectors that would be four warps and 10 cycles (the data pipe again);
// there a lane holds two lobes and shares their d and w, 11 cycles, and the
// two warps saved produce (30.5 against 36 cycles per sample and pass in a
// leaf of 30 lobes that no other block helps, before the producers' packed
// arithmetic).  The sum of a_k w multiplies by
// a row of ones, (1 a) w, which keeps its bits and the warp's lanes alike.
// Sixteen samples per turn, in four groups of four: a group's products are
// formed, its registers take the loads of the group four further on, then
// the products are added, so that a load has three groups of additions (50
// cycles) to arrive.  The products of two samples share one packed multiply
// (each component rounded as its own multiply).  The last turn's loads run up
// to 16 floats past the row; their values are not used.  The loop is inlined
// into the consumer's chunk loop and works on 32-bit shared-memory addresses.
__device__ __forceinline__ void add4(float &acc, float4 v) {
  acc += v.x;
  acc += v.y;
  acc += v.z;
  acc += v.w;
}
__device__ __forceinline__ float4 chain_terms(float4 a, float4 d, float4 w) {
  const float2 p0 = mul2(mul2(make_float2(d.x, d.y), make_float2(a.x, a.y)), make_float2(w.x, w.y));
  const float2 p1 = mul2(mul2(make_float2(d.z, d.w), make_float2(a.z, a.w)), make_float2(w.z, w.w));
  return make_float4(p0.x, p0.y, p1.x, p1.y);
}
// Rows start at 32-bit shared addresses A0 (A1: the second lobe's), D, W
// (bytes); n16 samples, a multiple of 16 (past the leaf's last sample the
// rows hold zeros).
template <bool kTwo>
__device__ __forceinline__ float2 chain_rows(uint32_t A0, uint32_t A1, uint32_t D, uint32_t W, int n16, float2 acc) {
  float4 a[4], b[4], d[4], w[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    a[g] = lds4(A0 + 16 * g);
    if (kTwo) b[g] = lds4(A1 + 16 * g);
    d[g] = lds4(D + 16 * g);
    w[g] = lds4(W + 16 * g);
  }
#pragma unroll 1
  for (int s = 0; s < n16; s += 16) {
    A0 += 64;
    A1 += 64;
    D += 64;
    W += 64;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float4 p = chain_terms(a[g], d[g], w[g]);
      a[g] = lds4(A0 + 16 * g);
      if (kTwo) {
        const float4 q = chain_terms(b[g], d[g], w[g]);
        b[g] = lds4(A1 + 16 * g);
        d[g] = lds4(D + 16 * g);
        w[g] = lds4(W + 16 * g);
        acc.x += p.x;
        acc.y += q.x;
        acc.x += p.y;
        acc.y += q.y;
        acc.x += p.z;
        acc.y += q.z;
        acc.x += p.w;
        acc.y += q.w;
      } else {
        d[g] = lds4(D + 16 * g);
        w[g] = lds4(W + 16 * g);
        add4(acc.x, p);
      }
    }
  }
  return acc;
}
__device__ __forceinline__ float value_rows(uint32_t R, int n16, float acc) {
  float4 a[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) a[g] = lds4(R + 16 * g);
#pragma unroll 1
  for (int s = 0; s < n16; s += 16) {
    R += 64;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float4 p = a[g];
      a[g] = lds4(R + 16 * g);
      add4(acc, p);
    }
  }
  return acc;
}
// The chains of consumer thread c: lane 8 q + j of chain warp v holds lobe
// 8 v + j, with four lobe vectors lobes 16 v + j and 16 v + 8 + j; q = 0 is the
// sum of a_k w, q = 1..3 of (d_q a_k) w.  Lanes 0-4 of the last warp hold the
// five per-sample rows (kind 2; the other lanes repeat the last of them).
struct ChainRole {
  int kind, k, q;  // 0: lobes k and k + 8; 1: lobe k; 2: row k
};
__device__ __forceinline__ ChainRole chain_role(const EStepShape &e, int c) {
  const int cw = c >> 5, lane = c & 31;
  if (cw + 1 == e.consWarps) return ChainRole{2, min(lane, 4), 0};
  return e.cnt == 4 ? ChainRole{0, 2 * cw * kLanes + (lane & 7), lane >> 3}
                    : ChainRole{1, cw * kLanes + (lane & 7), lane >> 3};
}
__device__ __forceinline__ void estep_chunk_chain(const EmShared &S, const float *B, const EStepShape &e,
                                                  const ChainRole &role, int n16, float2 &acc) {
  const int Kp = e.Kp;
  const uint32_t base = smem_u32(B), row = uint32_t(e.RS) * 4u;
  if (role.kind != 2) {
    const uint32_t X = base + uint32_t(Kp) * row, W = X + 3u * row;
    // the row of ones starts four banks after the z row, so the four
    // direction rows of a warp's load lie in distinct banks
    const uint32_t ones = smem_u32(S.ones);
    const uint32_t D = role.q == 0 ? ones + ((X + 3u * row - ones) & 127u) : X + uint32_t(role.q - 1) * row;
    const uint32_t A = base + uint32_t(role.k) * row;
    if (role.kind == 0) acc = chain_rows<true>(A, A + uint32_t(kLanes) * row, D, W, n16, acc);
    else acc = chain_rows<false>(A, A, D, W, n16, acc);
  } else {
    acc.x = value_rows(base + uint32_t(Kp + 4 + role.k) * row, n16, acc.x);
  }
}

// Barrier phase of chunk k: use k / stages of stage k % stages.
__device__ __forceinline__ uint32_t use_parity(const EmShared &S, const EStepShape &e, uint32_t k) {
  return (S.stageUses[k % uint32_t(e.stages)] + k / uint32_t(e.stages)) & 1u;
}
// Chunks that every consumer warp has added (they are added in order).
__device__ __forceinline__ uint32_t chunks_done(const EmShared &S, const EStepShape &e) {
  const volatile uint32_t *d = S.warpDone;
  uint32_t m = d[0];
  for (int w = 1; w < e.consWarps; ++w) m = min(m, d[w]);
  return m;
}

// Consumer warps (threads [cons0, 512)): chunk k is added once stage
// k % stages is full; each warp then records its progress.
__device__ __forceinline__ float2 consume_estep(EmShared &S, const EStepShape &e, uint32_t N, uint32_t count) {
  const int r = int(threadIdx.x) - e.cons0;
  const ChainRole role = chain_role(e, r);
  float2 acc = make_float2(0.0f, 0.0f);
  const int lane = int(threadIdx.x & 31);
  long long waited = 0;
  for (uint32_t k = 0; k < N; ++k) {
    const int st = int(k % uint32_t(e.stages));
    const long long w0 = clock64();
    if (!mbar_wait(&S.full[st], use_parity(S, e, k), &S.abortAt, k, S.err)) break;
    waited += clock64() - w0;
    const int n = int(min(uint32_t(e.C), count - chunk_begin(e, k)));
    estep_chunk_chain(S, S.pbuf + st * e.stageFloats, e, role, (n + 15) & ~15, acc);
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();  // this warp's reads of the stage come first
      reinterpret_cast<volatile uint32_t *>(S.warpDone)[r >> 5] = k + 1u;
    }
  }
  if (r == 0) S.prof.cycWaitE += uint64_t(waited);
  return acc;
}

// Waits until the consumers are done with chunk `need - 1` (bounded).
__device__ void wait_done(const EmShared &S, const EStepShape &e, uint32_t need) {
  unsigned long long t0 = 0;
  for (uint32_t it = 0; chunks_done(S, e) < need; ++it) {
    __nanosleep(64);
    if ((it & 31) == 31) {
      if (has_error(S.err)) return;
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitNs) {
        set_error(S.err, kErrSlotWait);
        return;
      }
    }
  }
  __threadfence_block();
}

// Loader warp: the chunks of the pass, 32 at a time.  A chunk is settled
// when this block's producers took it (they fill its stage) or when its ring
// slot holds it and its stage is free (then a bulk copy brings it in, also
// ahead of a late chunk); the settled count advances in order.  Ring slots are handed back as the copies land (all of them at the
// end of the pass).
__device__ void load_chunks(EmShared &S, const EStepShape &e, uint32_t N, uint32_t seqBase) {
  Board &b = *S.board;
  const int lane = int(threadIdx.x & 31);
  const uint32_t bytes = uint32_t(e.stageFloats) * 4u;
  const uint32_t stages = uint32_t(e.stages);
  uint32_t issued = 0, released = 0;
  unsigned handled = 0;  // bit i: chunk issued + i is settled (own, or its copy issued)
  unsigned long long t0 = 0;
  while (issued < N) {
    const uint32_t done = chunks_done(S, e);
    // a chunk's ring slot is free once its copy has landed (its stage's
    // barrier phase completed); stages of chunks past `done` are not reused
    // yet, so their phases are still the ones to test
    uint32_t rel = released > done ? released : done;
    while (rel < issued && mbar_test_wait(&S.full[rel % stages], use_parity(S, e, rel))) ++rel;
    if (rel > released) {
      if (lane == 0) st_release(&b.consumed, seqBase + rel);
      released = rel;
    }
    const uint32_t j = issued + uint32_t(lane);
    bool ok = (handled >> lane) & 1u, copy = false;
    if (!ok && j < N && j < done + stages) {  // stage j % stages is free
      const uint32_t seq = seqBase + j + 1u;
      if (reinterpret_cast<volatile uint32_t *>(S.own)[j & 63u] == seq) ok = true;
      else if (ld_relaxed(&b.ready[(seqBase + j) % uint32_t(e.slots)]) == seq) ok = copy = true;
    }
    const unsigned okMask = __ballot_sync(0xFFFFFFFFu, ok);
    const uint32_t prefix = okMask == 0xFFFFFFFFu ? 32u : uint32_t(__ffs(~okMask)) - 1u;  // settled from `issued` on
    // copies may be issued out of order (only the summing is in order): a
    // chunk that is ready behind a late one is copied now
    if (copy) {
      // the relaxed read saw the producer's release: acquire before the copy
      fence_acquire();
      fence_proxy_async();
      const int st = int(j % stages);
      mbar_expect_tx(&S.full[st], bytes);
      bulk_load(S.pbuf + st * e.stageFloats, S.ring + size_t((seqBase + j) % uint32_t(e.slots)) * e.stageFloats,
                bytes, &S.full[st]);
    }
    issued += prefix;
    handled = prefix >= 32u ? 0u : (okMask >> prefix);
    if (prefix == 0) {
      if (has_error(S.err)) {
        if (lane == 0) S.abortAt = issued;
        return;
      }
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitNs) {
        if (lane == 0) {
          set_error(S.err, kErrChunkWait);
          S.abortAt = issued;
        }
        return;
      }
      __nanosleep(200);
    } else {
      t0 = 0;
    }
    __syncwarp();
  }
}

// This block's producers (threads [0, P)): take chunks from their own board,
// write each into its stage once the consumers are done with the stage's
// previous chunk, and complete the stage's full barrier.  Producing a sample
// costs the SM several times the issue slots of adding it, so the producers
// step back while helpers supply the consumers: when the chunks they take
// are not consecutive (other blocks are taking chunks too), they take the
// next one only once the board's next free chunk is within `stages` of the
// consumers; while they are alone, the next grab overlaps the current
// chunk's production.
__device__ int take_own_chunk(EmShared &S, const EStepShape &e, Board &b, uint32_t gen) {
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    if (has_error(S.err)) return -1;
    const unsigned long long w = ld_relaxed64(&b.grab);
    if (grab_gen(w) != gen || grab_next(w) >= grab_chunks(w)) return -1;  // none left
    if (grab_next(w) < chunks_done(S, e) + uint32_t(e.stages)) {
      const unsigned long long w2 = atomicAdd(&b.grab, 1ull);
      return (grab_gen(w2) == gen && grab_next(w2) < grab_chunks(w2)) ? int(grab_next(w2)) : -1;
    }
    __nanosleep(256);
    if ((it & 15) == 15) {
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitNs) {
        set_error(S.err, kErrChunkWait);
        return -1;
      }
    }
  }
}
__device__ void produce_own(EmShared &S, const EStepShape &e, const LeafSamples &L, uint32_t seqBase) {
  Board &b = *S.board;
  const int t = threadIdx.x;
  const uint32_t gen = S.gen;  // read by thread 0 only, which wrote it
  bool alone = true;           // thread 0: the last two chunks taken were consecutive
  if (t == 0) {
    const unsigned long long w = atomicAdd(&b.grab, 1ull);
    S.hgrab[0] = (!has_error(S.err) && grab_gen(w) == gen && grab_next(w) < grab_chunks(w)) ? int(grab_next(w)) : -1;
  }
  uint32_t made = 0;
  for (uint32_t i = 0;; ++i) {
    if (t == 0) {
      const int c0 = S.hgrab[i & 1u];
      if (c0 >= 0) {
        // mark the chunk as this block's only once its stage is free: it is
        // then within `stages` chunks of the consumers, so the marker's slot
        // (chunk - 64) has been settled and consumed long ago
        const uint32_t k = uint32_t(c0);
        if (k >= uint32_t(e.stages)) wait_done(S, e, k - uint32_t(e.stages) + 1u);
        reinterpret_cast<volatile uint32_t *>(S.own)[k & 63u] = seqBase + k + 1u;
      }
    }
    bar_named(3, e.P);
    const int chunk = S.hgrab[i & 1u];
    if (chunk < 0) break;
    ++made;
    const uint32_t k = uint32_t(chunk);
    const int st = int(k % uint32_t(e.stages));
    unsigned long long w = 0;
    const bool early = t == 0 && alone;
    if (early) w = atomicAdd(&b.grab, 1ull);
    produce_estep_chunk(S, e, L.dirw, L.count, k, S.pbuf + st * e.stageFloats, t, e.P);
    bar_named(3, e.P);
    if (t == 0) {
      mbar_arrive(&S.full[st]);
      int nextChunk;
      if (early) {
        nextChunk = (grab_gen(w) == gen && grab_next(w) < grab_chunks(w)) ? int(grab_next(w)) : -1;
        alone = nextChunk == chunk + 1;
      } else {
        nextChunk = take_own_chunk(S, e, b, gen);
      }
      S.hgrab[(i + 1u) & 1u] = nextChunk;
    }
  }
  if (t == 0) S.prof.chunksOwn += made;
}

// E-step over all samples into S.cur, S.ll and S.un (WEMFactory.h:847-892).
__device__ void pass_estep(EmShared &S, const LeafSamples &L) {
  const int tid = threadIdx.x;
  const int cnt = vec_count(int(S.vmm.K));
  const EStepShape e = estep_shape(cnt, S.tune);
  const int Kp = e.Kp;
  uint32_t N = L.count == 0 ? 0u : chunk_count(e, L.count);
  if (N > kMaxSharedChunks) {
    if (tid == 0) set_error(S.err, kErrLeafTooLarge);
    N = 0;
  }
  if (tid == 0) {
    S.un = Unassigned{0.f, 0.f, 0.f, 0.f};
    suff_clear(S.cur, S.vmm.K);
    S.cur.K = S.vmm.K;
    S.cur.numSamples = float(L.count);
    S.abortAt = has_error(S.err) ? 0u : 0xFFFFFFFFu;
  }
  if (tid < kEmThreads / 32) S.warpDone[tid] = 0;
  pack_pairs(S, Kp);
  __syncthreads();
  const uint32_t seqBase = S.seqBase;
  if (tid == 0) {  // publish the pass on the board
    Board &b = *S.board;
    const uint32_t gen = S.gen % kGrabGenMask + 1u;
    S.gen = gen;
    BoardParams &bp = b.params[gen & 1u];
    for (int i = 0; i < pair_at(Kp); ++i) bp.lobeP[i] = S.lobeP[i];
    bp.dirw = L.dirw;
    bp.count = L.count;
    bp.seqBase = seqBase;
    bp.cnt = uint32_t(cnt);
    __threadfence();
    atomicExch(&b.grab, grab_word(gen, N, 0));
  }
  float2 acc = make_float2(0.0f, 0.0f);
  const long long t0 = clock64();
  if (tid < e.P) produce_own(S, e, L, seqBase);
  else if (tid < e.cons0) load_chunks(S, e, N, seqBase);
  else acc = consume_estep(S, e, N, L.count);
  const long long cyc = clock64() - t0;
  if (tid == 0) S.prof.cycProdE += uint64_t(cyc);
  if (tid == e.cons0) S.prof.cycConsE += uint64_t(cyc);
  __syncthreads();
  if (tid >= e.cons0) {
    const ChainRole role = chain_role(e, tid - e.cons0);
    if (role.kind != 2) {
      float *sum = role.q == 0 ? S.cur.w : role.q == 1 ? S.cur.dx : role.q == 2 ? S.cur.dy : S.cur.dz;
      sum[role.k] = acc.x;
      if (role.kind == 0) sum[role.k + kLanes] = acc.y;
    } else if ((tid & 31) < 5) {
      const int x = role.k;
      if (x == 0) S.ll = acc.x;
      else if (x == 1) S.un.sw = acc.x;
      else if (x == 2) S.un.dx = acc.x;
      else if (x == 3) S.un.dy = acc.x;
      else S.un.dz = acc.x;
    }
  }
  if (tid == 0) {
    S.prof.chunks += N;
    for (int st = 0; st < e.stages; ++st)
      S.stageUses[st] += N > uint32_t(st) ? (N - uint32_t(st) + uint32_t(e.stages) - 1u) / uint32_t(e.stages) : 0u;
    S.seqBase = seqBase + N;
    st_release(&S.board->consumed, seqBase + N);
  }
  __syncthreads();
}

// A block without leaves produces chunks for other blocks' E-step passes:
// it picks the board with the most chunks left (among boards with fewer than
// EmTuning::maxHelpers helpers) and takes chunks from it while
// it has any (loading the pass parameters when the generation changes).  It
// leaves once every leaf of the launch is finished (or the launch failed).
__device__ void help_others(EmShared &S, Board *boards, float *rings, const uint32_t *finished, uint32_t numTasks) {
  const int tid = threadIdx.x;
  const int nb = int(gridDim.x);
  int cachedBoard = -1;
  uint32_t cachedGen = 0;
  for (;;) {
    // scan: the board with the most chunks left
    uint32_t bestRem = 0;
    int best = -1;
    for (int i = tid; i < nb; i += kEmThreads) {
      const unsigned long long w = ld_relaxed64(&boards[i].grab);
      const uint32_t n = grab_chunks(w), nx = grab_next(w);
      const bool open = ld_relaxed(&boards[i].helpers) < uint32_t(S.tune.maxHelpers);
      const uint32_t rem = (grab_gen(w) != 0 && nx < n && open) ? n - nx : 0u;
      if (rem > bestRem) {
        bestRem = rem;
        best = i;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      const uint32_t r = __shfl_down_sync(0xFFFFFFFFu, bestRem, off);
      const int i = __shfl_down_sync(0xFFFFFFFFu, best, off);
      if (r > bestRem) {
        bestRem = r;
        best = i;
      }
    }
    if ((tid & 31) == 0) {
      S.scanRem[tid >> 5] = bestRem;
      S.scanIdx[tid >> 5] = best;
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t r = 0;
      int bi = -1;
      for (int w = 0; w < kEmThreads / 32; ++w)
        if (S.scanRem[w] > r) {
          r = S.scanRem[w];
          bi = S.scanIdx[w];
        }
      S.helpBoard = bi;
      S.helpExit = has_error(S.err) || (bi < 0 && ld_acquire(finished) >= numTasks);
    }
    __syncthreads();
    if (S.helpExit) return;
    const int bi = S.helpBoard;
    if (bi < 0) {
      __nanosleep(1000);
      continue;
    }
    Board &b = boards[bi];
    // attach to the board while it has fewer than maxHelpers helpers: with
    // at most one chunk held per helper, the chunks taken stay close to the
    // ring's free slots, and the other helpers stay free for other boards
    if (tid == 0) {
      const uint32_t before = atomicAdd(&b.helpers, 1u);
      S.helpExit = before < uint32_t(S.tune.maxHelpers) ? 0 : 1;
      if (before >= uint32_t(S.tune.maxHelpers)) atomicSub(&b.helpers, 1u);
    }
    __syncthreads();
    if (S.helpExit) {
      __syncthreads();
      __nanosleep(500);
      continue;
    }
    if (tid == 0) S.hasNext = 0;
    for (int tries = 0;;) {
      if (tid == 0) {
        if (S.hasNext) {  // taken while the last chunk was produced
          S.grabbed = S.nextGrabbed;
          S.grabGen = S.nextGen;
          S.grabExact = S.nextExact;
          S.hasNext = 0;
        } else {
          uint32_t g = 0;
          int x = 0;
          S.grabbed = helper_take(S, b, bi == cachedBoard, cachedGen, g, x);
          if (S.grabbed != -2 && S.grabbed != -1) S.grabGen = g;
          S.grabExact = x;
        }
      }
      __syncthreads();
      const int chunk = S.grabbed;
      const uint32_t gen = S.grabGen;
      if (chunk == -2) {
        __syncthreads();  // everyone has read S.grabbed before thread 0 rewrites it
        if (++tries > 64) break;  // look at the other boards again
        __nanosleep(200);
        continue;
      }
      if (chunk < 0) break;
      tries = 0;
      if (bi != cachedBoard || gen != cachedGen) {
        // the generation was published (atomic exchange) after its parameters
        if (tid == 0) __threadfence();
        __syncthreads();
        const BoardParams &src = b.params[gen & 1u];
        for (int i = tid; i < kPairEntries; i += kEmThreads) S.lobeP[i] = __ldcg(&src.lobeP[i]);
        if (tid == 0) {
          S.hp.dirw = reinterpret_cast<const float4 *>(__ldcg(reinterpret_cast<const unsigned long long *>(&src.dirw)));
          S.hp.count = __ldcg(&src.count);
          S.hp.seqBase = __ldcg(&src.seqBase);
          S.hp.cnt = __ldcg(&src.cnt);
        }
        __syncthreads();
        cachedBoard = bi;
        cachedGen = gen;
      }
      const EStepShape e = estep_shape(int(S.hp.cnt), S.tune);
      produce_for(S, b, rings + size_t(bi) * kRingFloats, e, S.hp.dirw, S.hp.count, S.hp.seqBase, uint32_t(chunk),
                  S.grabExact != 0, cachedGen);
      __syncthreads();
    }
    if (tid == 0) atomicSub(&b.helpers, 1u);
  }
}

// init/updateComponentDistances (WEMFactory.h:1199-1326)
__device__ void pass_distances(EmShared &S, const LeafSamples &L, bool init) {
  const int tid = threadIdx.x;
  const int cnt = vec_count(int(S.vmm.K));
  const int Kp = cnt * kLanes;
  pack_pairs(S, Kp);
  if (tid < Kp) {
    const float w = uint32_t(tid) < S.vmm.K ? S.vmm.w[tid] : 1.0f;  // the sums of lobes past the last are not used
    S.lobeW[tid] = make_float2(w, (w >= 1e-8f && w <= 1e8f) ? rcp_newton(w) : 0.0f);
  }
  __syncthreads();
  switch (cnt) {
    case 1: run_distance<1>(S, L); break;
    case 2: run_distance<2>(S, L); break;
    case 3: run_distance<3>(S, L); break;
    default: run_distance<4>(S, L); break;
  }
  // sums over rcp(distance) in xch[0], over 1 in xch[1]
  if (tid == 0) {
    VMMState &v = S.vmm;
    SuffState &s = S.suff;
    int cc = vec_count(int(v.K)), rem = int(v.K % kLanes);
    for (int kk = 0; kk < cc * kLanes; ++kk) {
      float bd = S.xch[0][kk], bw = S.xch[1][kk];
      if (init) {
        s.dw[kk] = bw;
        v.dist[kk] = s.dw[kk] / bd;
      } else {
        float inv = bd;
        inv += v.dist[kk] > 0.0f ? (s.dw[kk] / v.dist[kk]) : 0.0f;
        s.dw[kk] += bw;
        v.dist[kk] = s.dw[kk] / inv;
      }
    }
    if (rem > 0)
      for (int i = rem; i < kLanes; ++i) { v.dist[(cc - 1) * kLanes + i] = 0.0f; s.dw[(cc - 1) * kLanes + i] = 0.0f; }
  }
  __syncthreads();
}

// UpdateSplitStatistics (Splitter.h:439-523) into sp (S.split or S.lsplit).
__device__ void pass_split_stats(EmShared &S, const LeafSamples &L, SplitState &sp) {
  const int tid = threadIdx.x;
  const int cnt = vec_count(int(sp.K));
  const int Kp = cnt * kLanes;
  if (2 * tid < Kp) {
    const int k = 2 * tid;
    const Frame f0 = inverse_of(frame_of(mk(S.vmm.mx[k], S.vmm.my[k], S.vmm.mz[k]), true));
    const Frame f1 = inverse_of(frame_of(mk(S.vmm.mx[k + 1], S.vmm.my[k + 1], S.vmm.mz[k + 1]), true));
    float4 *o = S.frameP + pair_at(k);
    o[0] = make_float4(f0.vx.x, f1.vx.x, f0.vy.x, f1.vy.x);
    o[1] = make_float4(f0.vz.x, f1.vz.x, f0.vx.y, f1.vx.y);
    o[2] = make_float4(f0.vy.y, f1.vy.y, f0.vz.y, f1.vz.y);
  }
  pack_pairs(S, Kp);
  __syncthreads();
  switch (cnt) {
    case 1: run_split<1>(S, L, sp); break;
    case 2: run_split<2>(S, L, sp); break;
    case 3: run_split<3>(S, L, sp); break;
    default: run_split<4>(S, L, sp); break;
  }
}

// updateMixture / partialUpdateMixture (WEMFactory.h:751-844).  prev is the
// "previous" statistics (S.suff or S.temp); partial uses S.mask.
__device__ int em_loop(EmShared &S, const LeafSamples &L, SuffState &prev, bool partial, const FieldConfig &cfg) {
  const int tid = threadIdx.x;
  __shared__ float prevLL, invPrevLL;
  if (tid == 0) {
    suff_clear(S.cur, kMaxK);
    S.cur.overallNumSamples = 0.0f;
    S.iterations = 0;
    S.loopFlag = 1;
    prevLL = 0.0f;
    invPrevLL = 1.0f;
  }
  __syncthreads();
  while (S.loopFlag) {
    PGL_PROF_BEGIN(t0)
    pass_estep(S, L);
    PGL_PROF_END(t0, cycEstep)
    PGL_PROF_BEGIN(t1)
    if (tid < 32) {  // the M-step by warp 0, lane k on lobe k
      if (tid == 0) {
        S.prof.estepPasses++;
        S.prof.estepLobes += S.vmm.K;
        if (S.un.sw > 0.0f && S.cur.K < kMaxK) {  // handleUnassignedSampleStats (WEMFactory.h:731-748)
          int t = int(S.cur.K);
          S.cur.K++;
          S.cur.w[t] = S.un.sw; S.cur.dx[t] = S.un.dx; S.cur.dy[t] = S.un.dy; S.cur.dz[t] = S.un.dz;
          prev.K++;
          prev.w[t] = 0.0f; prev.dx[t] = prev.dy[t] = prev.dz[t] = 0.0f;
          S.vmm.K++;
          if (partial) S.mask[S.vmm.K - 1] = 1;
        }
      }
      __syncwarp();
      suff_normalize_warp(S.cur, S.cur.numSamples);
      map_step_warp(S.vmm, S.cur, prev, cfg, partial ? S.mask : nullptr);
    }
    if (tid == 0) {
      S.iterations++;
      bool converged = false;
      if (S.iterations > 1) {
        float rel = fabsf(S.ll - prevLL) * invPrevLL;
        if (rel < cfg.convergence) converged = true;
        prevLL = S.ll;
        invPrevLL = 1.0f / fabsf(S.ll);
      }
      S.loopFlag = (!converged && uint32_t(S.iterations) < cfg.maxIter) ? 1 : 0;
    }
    PGL_PROF_END(t1, cycMstep)
    __syncthreads();
  }
  if (tid == 0) suff_add(prev, S.cur);
  __syncthreads();
  return S.iterations;
}

// getSplitCandidates (Splitter.h:1103-1117) by one warp: descending chi-square,
// equal values keep index order (values without an order, NaN, as the
// insertion sort of one thread leaves them).
__device__ void sort_candidates(EmShared &S, const SplitState &sp) {
  const int n = int(sp.K), lane = threadIdx.x & 31;
  const unsigned full = 0xFFFFFFFFu;
  const float c = lane < n ? sp.chi2[lane] : 0.0f;
  if (__any_sync(full, c != c)) {
    if (lane == 0) {
      for (int i = 0; i < n; ++i) { S.candIdx[i] = i; S.candChi[i] = sp.chi2[i]; }
      for (int i = 1; i < n; ++i) {
        int ci = S.candIdx[i];
        float cv = S.candChi[i];
        int j = i - 1;
        while (j >= 0 && cv > S.candChi[j]) { S.candIdx[j + 1] = S.candIdx[j]; S.candChi[j + 1] = S.candChi[j]; --j; }
        S.candIdx[j + 1] = ci;
        S.candChi[j + 1] = cv;
      }
    }
  } else {
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const float o = __shfl_sync(full, c, j);
      rank += (o > c || (o == c && j < lane)) ? 1 : 0;
    }
    if (lane < n) {
      S.candIdx[rank] = lane;
      S.candChi[rank] = c;
    }
  }
  if (lane == 0) S.numCands = n;
  __syncwarp();
}
// Splits the candidates above the threshold in order while there are slots
// (Splitter.h:293-356, 364-420), by one warp, a lane per candidate: a split reads
// its own component only and takes the slot behind the splits before it.  One
// thread took 60,000 to 190,000 cycles per region and Update, a twentieth of a
// small region's time.  Returns the splits made; tried: the candidates
// considered.
__device__ int split_candidates(EmShared &S, SplitState &sp, SuffState &suff, int n, const FieldConfig &cfg, int &tried) {
  VMMState &v = S.vmm;
  const int lane = threadIdx.x & 31, K = int(v.K);
  const unsigned full = 0xFFFFFFFFu;
  const bool wanted = lane < n && S.candChi[lane] > cfg.splitThreshold;
  const int idx = wanted ? S.candIdx[lane] : 0;
  SplitLobes o;
  bool ok = wanted && split_component(v, sp, idx, cfg, o);
  const int slot = K + __popc(__ballot_sync(full, ok) & ((1u << lane) - 1u));  // K when its turn comes
  const bool considered = wanted && slot < int(kMaxK);
  ok = ok && considered;
  if (ok) {
    vmm_split(v, idx, slot, o.w, o.w, o.m0, o.m1, o.mc0, o.mc1);
    suff_split(suff, idx, slot, o.m0, o.m1, o.mc0, o.mc1);
    split_zero_lane(sp, idx);
    split_zero_lane(sp, slot);
  }
  if (considered) {
    S.mask[idx] = 1;
    S.mask[ok ? slot : slot - 1] = 1;  // the last component after its turn
  }
  const int made = __popc(__ballot_sync(full, ok));
  tried = __popc(__ballot_sync(full, considered));
  __syncwarp();
  if (made > 0) {
    if (lane == 0) {
      v.K = uint32_t(K + made);
      sp.K = uint32_t(K + made);
      suff.K += uint32_t(made);
    }
    if (lane < vec_count(K + made) * kLanes) {  // vmm_calc_norm
      v.e2k[lane] = fexp(-2.0f * v.kappa[lane]);
      const float nrm = v.kappa[lane] / (kTwoPiF * (1.0f - v.e2k[lane]));
      v.norm[lane] = v.kappa[lane] > 0.0f ? nrm : kInv4Pi;
    }
  }
  __syncwarp();
  return made;
}

// PerformMerging (Merger.h:67-89, 218-279): all pair costs in parallel, then
// the first minimum in (i, j) scan order below the threshold, as the smallest
// (cost, i, j) over the block's threads.  A region's merging was bound by the
// costs' double-precision functions and their table searches and by one
// thread's scan of the pairs: 1.3 M cycles per region with 23 to 30 lobes, 0.3 M
// without those, 0.19 M with the parts of a cost spread over threads (fourth
// frame of 2,097,152 samples, whose EM launch took 4.3, 3.1 and 2.0 ms with the
// other steps of the time).
__device__ int perform_merging(EmShared &S, const FieldConfig &cfg) {
  const int tid = threadIdx.x;
  __shared__ int mergeAgain, total, lastI, lastJ;
  __shared__ unsigned long long warpBest[kEmThreads / 32];
  if (tid == 0) { total = 0; mergeAgain = S.vmm.K > cfg.laneWidth ? 1 : 0; lastI = -1; lastJ = -1; }
  __syncthreads();
  while (mergeAgain) {
    const int K = int(S.vmm.K);
    if (lastI < 0) {  // every pair
      const int pairs = K * (K - 1) / 2;
      for (int first = 0; first < pairs; first += kMergePairs) {
        const int nP = min(pairs - first, kMergePairs);
        for (int q = tid; q < nP; q += kEmThreads) {
          // the pair's (i, j), i < j
          int i = 0, rem = first + q;
          while (rem >= K - 1 - i) { rem -= K - 1 - i; ++i; }
          S.merge.i[q] = uint8_t(i);
          S.merge.j[q] = uint8_t(i + 1 + rem);
        }
        __syncthreads();
        merge_costs(S, nP, first == 0 ? 0xFFFFFFFFu >> (kMaxK - K) : 0u);
        __syncthreads();
      }
    } else {
      // after merging lastJ into lastI (and moving the last component into
      // slot lastJ) only the pairs with those two slots have new operands; a
      // pair's cost depends on its two components alone, so the others keep
      // the bits a full recomputation would give
      const int moved = lastJ < K ? 1 : 0;  // lastJ was not the last slot
      for (int t = tid; t < (1 + moved) * K; t += kEmThreads) {
        const int a = t < K ? lastI : lastJ, b = t < K ? t : t - K;
        const bool none = b == a || (a == lastJ && b == lastI);  // (lastI, lastJ) is in the first row
        S.merge.i[t] = none ? uint8_t(255) : uint8_t(min(a, b));
        S.merge.j[t] = uint8_t(max(a, b));
      }
      __syncthreads();
      merge_costs(S, (1 + moved) * K, 1u << lastI | (moved ? 1u << lastJ : 0u));
      __syncthreads();
    }
    // the reference's row-major double loop (Merger.h:67-90) keeps the first of equal
    // costs; both zeros are equal
    unsigned long long best = ~0ull;
    for (int t = tid; t < K * kMaxK; t += kEmThreads) {
      const int i = t / kMaxK, j = t % kMaxK;
      if (j <= i || j >= K) continue;
      const float cost = S.cost[i][j];
      if (cost < cfg.mergeThreshold && cost < FLT_MAX && S.split.n[i] > 0.0f && S.split.n[j] > 0.0f) {
        const unsigned long long key =
            (static_cast<unsigned long long>(float_key(cost == 0.0f ? 0.0f : cost)) << 32) | uint32_t(t);
        best = key < best ? key : best;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long o = __shfl_down_sync(0xFFFFFFFFu, best, off);
      best = o < best ? o : best;
    }
    if ((tid & 31) == 0) warpBest[tid >> 5] = best;
    __syncthreads();
    if (tid == 0 || tid == 32) {
      best = warpBest[0];
      for (int w = 1; w < kEmThreads / 32; ++w) best = warpBest[w] < best ? warpBest[w] : best;
      const bool found = best != ~0ull;
      const int ci = int(uint32_t(best)) / kMaxK, cj = int(uint32_t(best)) % kMaxK;
      if (found && tid == 32) suff_merge(S.suff, ci, cj);
      if (found && tid == 0) {
        VMMState &v = S.vmm;
        V3 muI = mk(v.mx[ci], v.my[ci], v.mz[ci]), muJ = mk(v.mx[cj], v.my[cj], v.mz[cj]);
        float wI = v.w[ci], wJ = v.w[cj];
        vmm_merge(v, ci, cj);
        V3 muK = mk(v.mx[ci], v.my[ci], v.mz[ci]);
        split_merge_stats(S.split, ci, cj, wI, muI, wJ, muJ, v.w[ci], muK);
        total++;
        lastI = ci;
        lastJ = cj;
      }
      if (tid == 0) mergeAgain = (found && S.vmm.K > cfg.laneWidth) ? 1 : 0;
    }
    __syncthreads();
  }
  return total;
}

// PerformRecursiveSplitting (Splitter.h:293-356) with temp = copy of suff.
__device__ void recursive_splitting(EmShared &S, const LeafSamples &L, const FieldConfig &cfg) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.temp = S.suff;
    S.splitCount = -1;
  }
  __syncthreads();
  while (S.vmm.K < kMaxK && S.splitCount != 0) {
    if (tid == 0) {
      S.splitCount = 0;
      split_clear(S.lsplit, kMaxK);
      split_clear(S.lsplit, S.vmm.K);
    }
    __syncthreads();
    {
      PGL_PROF_BEGIN(tp0)
      if (threadIdx.x == 0) { S.prof.splitPasses++; S.prof.splitLobes += S.lsplit.K; }
      pass_split_stats(S, L, S.lsplit);
      PGL_PROF_END(tp0, cycSplit)
    }
    if (tid < 32) {
      sort_candidates(S, S.lsplit);
      S.mask[tid] = 0;
      __syncwarp();
      int tried;
      const int made = split_candidates(S, S.lsplit, S.temp, int(S.vmm.K), cfg, tried);
      if (tid == 0) {
        S.splitCount += made;
        if (S.splitCount > 0) suff_clear(S.temp, S.vmm.K);
      }
    }
    __syncthreads();
    if (S.splitCount > 0) {
      em_loop(S, L, S.temp, true, cfg);
      if (tid == 0) {
        S.suff.K = S.vmm.K;
        suff_masked_replace(S.suff, S.mask, S.temp);
      }
      __syncthreads();
    }
  }
}

// Fit (first frame) of one leaf (ASMF.h:303-347)
__device__ void asm_fit(EmShared &S, const LeafSamples &L, const FieldConfig &cfg, const float *uniformDirs) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    suff_clear(S.suff, cfg.initK);
    split_clear(S.split, cfg.initK);
    vmm_init_uniform(S.vmm, int(cfg.initK), cfg.initKappa, uniformDirs);
    suff_clear(S.suff, cfg.initK);
    S.suff.normalized = 1;
  }
  __syncthreads();
  S.report.emIterations += em_loop(S, L, S.suff, false, cfg);
  {
    PGL_PROF_BEGIN(tp0)
    if (threadIdx.x == 0) { S.prof.distPasses++; S.prof.distLobes += S.vmm.K; }
    pass_distances(S, L, true);
    PGL_PROF_END(tp0, cycDist)
  }
  if (cfg.useSplitMerge) {
    if (tid == 0) S.mcEstimate = S.suff.sumWeights / S.suff.numSamples;
    __syncthreads();
    recursive_splitting(S, L, cfg);
    if (tid == 0) split_clear(S.split, S.vmm.K);
    __syncthreads();
    {
      PGL_PROF_BEGIN(tp1)
      if (threadIdx.x == 0) { S.prof.splitPasses++; S.prof.splitLobes += S.split.K; }
      pass_split_stats(S, L, S.split);
      PGL_PROF_END(tp1, cycSplit)
    }
    PGL_PROF_BEGIN(tm)
    int m = perform_merging(S, cfg);
    PGL_PROF_END(tm, cycMerge)
    if (tid == 0) S.report.merges += uint32_t(m);
  }
  {
    PGL_PROF_BEGIN(tp1)
    if (threadIdx.x == 0) { S.prof.distPasses++; S.prof.distLobes += S.vmm.K; }
    pass_distances(S, L, true);
    PGL_PROF_END(tp1, cycDist)
  }
}

// Update (later frames) of one leaf (ASMF.h:352-462)
__device__ void asm_update(EmShared &S, const LeafSamples &L, const FieldConfig &cfg, uint64_t &afterSplit,
                           uint64_t &afterMerge) {
  const int tid = threadIdx.x;
  __shared__ uint32_t prevK;
  __shared__ int doRefit;
  if (tid == 0) prevK = S.vmm.K;
  __syncthreads();
  S.report.emIterations += em_loop(S, L, S.suff, false, cfg);
  if (tid == 0 && prevK < S.vmm.K) S.split.K = S.vmm.K;
  __syncthreads();
  if (cfg.useSplitMerge) {
    if (tid == 0) {
      S.mcEstimate = S.suff.sumWeights / S.suff.numSamples;
      afterSplit += L.count;
      afterMerge += L.count;
    }
    __syncthreads();
    {
      PGL_PROF_BEGIN(tp2)
      if (threadIdx.x == 0) { S.prof.splitPasses++; S.prof.splitLobes += S.split.K; }
      pass_split_stats(S, L, S.split);
      PGL_PROF_END(tp2, cycSplit)
    }
    if (afterSplit >= uint64_t(int64_t(cfg.minSplit))) {
      if (tid < 32) {
        S.mask[tid] = 0;
        sort_candidates(S, S.split);
        int total;
        split_candidates(S, S.split, S.suff, S.numCands, cfg, total);
        if (tid == 0) {
          S.report.splits += uint32_t(total);
          doRefit = (total > 0 && cfg.partialReFit && uint64_t(L.count) >= uint64_t(int64_t(cfg.minRefit))) ? 1 : 0;
          if (doRefit) {
            S.temp = S.suff;
            suff_clear(S.temp, S.vmm.K);
          }
        }
      }
      __syncthreads();
      if (doRefit) {
        em_loop(S, L, S.temp, true, cfg);
        if (tid == 0) {
          S.suff.K = S.vmm.K;
          suff_masked_replace(S.suff, S.mask, S.temp);
          S.split.K = S.vmm.K;
        }
      }
      if (tid == 0) afterSplit = 0;
      __syncthreads();
    }
    if (afterMerge >= uint64_t(int64_t(cfg.minMerge))) {
      PGL_PROF_BEGIN(tm)
      int m = perform_merging(S, cfg);
      PGL_PROF_END(tm, cycMerge)
      if (tid == 0) { S.report.merges += uint32_t(m); afterMerge = 0; }
      __syncthreads();
    }
  }
  {
    PGL_PROF_BEGIN(tp2)
    if (threadIdx.x == 0) { S.prof.distPasses++; S.prof.distLobes += S.vmm.K; }
    pass_distances(S, L, false);
    PGL_PROF_END(tp2, cycDist)
  }
}

// Reprojection of a leaf's samples to the region's sample mean
// (WEMFactory.h:1151-1196); positions are not needed afterwards.
// WEMFactory::prepareSamples (WEMFactory.h:1183-1196): parallax-aware
// mixtures reproject the samples onto the region's mean; plain ones keep them
// (the distance passes still read each sample's distance).
__device__ void reproject_leaf(const LeafTask &t, float4 *pd, float4 *dirw, float *dist, bool parallax) {
  if (!parallax) {
    for (uint32_t i = threadIdx.x; i < t.count; i += blockDim.x) dist[t.begin + i] = pd[t.begin + i].w;
    return;
  }
  V3 var = mk(t.varOverN[0], t.varOverN[1], t.varOverN[2]);
  float minD = length(var);
  minD = 3.f * 3.f * sqrtf(minD);
  const V3 mean = mk(t.mean[0], t.mean[1], t.mean[2]);
  for (uint32_t i = threadIdx.x; i < t.count; i += blockDim.x) {
    uint32_t g = t.begin + i;
    float4 p = pd[g];
    float4 dw = dirw[g];
    float dd = p.w;
    if (isinf(dd) || !(dd > 0.0f)) { dist[g] = dd; continue; }
    float dm = fmaxf(minD, dd);
    V3 o = mk(p.x, p.y, p.z) + mk(dw.x, dw.y, dw.z) * dm;
    V3 nd = o - mean;
    float nl = length(nd);
    nd = nd / nl;
    dirw[g] = make_float4(nd.x, nd.y, nd.z, dw.w);
    dist[g] = nl;
  }
}

__global__ void __launch_bounds__(kEmThreads)
em_leaf_kernel(const LeafTask *tasks, uint32_t numTasks, unsigned int *queue, EmSides sides, LeafReport *reports,
               LeafProfile *profiles, Board *boards, float *rings, int *err, uint32_t *finished, EmTuning tune) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  EmShared &S = *reinterpret_cast<EmShared *>(smem_raw);
  __shared__ uint32_t taskId;
  __shared__ uint64_t afterSplit, afterMerge;
  for (int i = threadIdx.x; i < 2048; i += blockDim.x) S.rcpTab[i] = rcp_seed(uint32_t(i));
  for (int i = threadIdx.x; i < 64; i += blockDim.x) S.own[i] = 0;
  for (int i = threadIdx.x; i < kMaxChunk + 48; i += blockDim.x) S.ones[i] = 1.0f;
  if (threadIdx.x == 0) {
    S.board = boards + blockIdx.x;
    S.ring = rings + size_t(blockIdx.x) * kRingFloats;
    S.err = err;
    S.tune = tune;
    S.gen = 0;
    S.seqBase = 0;
    for (int i = 0; i < kMaxStages; ++i) {
      mbar_init(&S.full[i], 1);
      S.stageUses[i] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  // the plain form: block b fits region task b and exits (no queue, no help)
  const bool plain = tune.plainLaunches != 0;
  for (uint32_t round = 0;; ++round) {
    if (threadIdx.x == 0) taskId = plain ? (round == 0 ? blockIdx.x : numTasks) : atomicAdd(queue, 1u);
    __syncthreads();
    if (taskId >= numTasks) break;
    const LeafTask t = tasks[taskId];
    const EmSide &E = sides.side[(t.flags & kTaskVolume) ? 1 : 0];
    const FieldConfig &cfg = E.cfg;
    RegionDir &R = E.regions[t.region];
    // load the region's directional state
    {
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&R.vmm);
      uint32_t *dst = reinterpret_cast<uint32_t *>(&S.vmm);
      for (int i = threadIdx.x; i < int(sizeof(VMMState) / 4); i += blockDim.x) dst[i] = src[i];
      src = reinterpret_cast<const uint32_t *>(&R.suff);
      dst = reinterpret_cast<uint32_t *>(&S.suff);
      for (int i = threadIdx.x; i < int(sizeof(SuffState) / 4); i += blockDim.x) dst[i] = src[i];
      src = reinterpret_cast<const uint32_t *>(&R.split);
      dst = reinterpret_cast<uint32_t *>(&S.split);
      for (int i = threadIdx.x; i < int(sizeof(SplitState) / 4); i += blockDim.x) dst[i] = src[i];
    }
    const long long leafStart = clock64();
    if (threadIdx.x == 0) {
      S.prof = LeafProfile{};
      S.prof.count = t.count;
      S.prof.tBegin = global_ns();
      afterSplit = R.afterSplit;
      afterMerge = R.afterMerge;
      S.report = LeafReport{0, 0, 0, 0};
    }
    reproject_leaf(t, E.pd, E.dirw, E.dist, cfg.parallax != 0);
    __syncthreads();
    const bool fit = (t.flags & kTaskFit) != 0;
    if (!fit && (t.flags & kTaskDecay) && threadIdx.x == 0) {  // Field.h:457-461
      suff_decay(S.suff, cfg.decayOnSpatialSplit);
      split_decay(S.split, cfg.decayOnSpatialSplit);
    }
    __syncthreads();
    uint32_t valid = R.valid;
    if (t.count > 0) {
      LeafSamples L{E.dirw + t.begin, E.pdf + t.begin, E.dist + t.begin, t.count};
      if (fit) {
        asm_fit(S, L, cfg, E.uniformDirs);
        if (threadIdx.x < 32) valid = vmm_is_valid(S.vmm) ? 1u : 0u;
        if (threadIdx.x == 0) {
          S.vmm.pivot[0] = t.mean[0]; S.vmm.pivot[1] = t.mean[1]; S.vmm.pivot[2] = t.mean[2];
          afterSplit = 0;
          afterMerge = 0;
        }
      } else {
        if (threadIdx.x < 32 && cfg.parallax) {  // Field.h:476-482, a lane per lobe
          const V3 shift = mk(S.vmm.pivot[0] - t.mean[0], S.vmm.pivot[1] - t.mean[1], S.vmm.pivot[2] - t.mean[2]);
          const int k = threadIdx.x;
          if (k < vec_count(int(S.vmm.K)) * kLanes) {
            suff_parallax_shift(S.suff, S.vmm, shift, k);
            vmm_parallax_shift(S.vmm, shift, k);
          }
          __syncwarp();
          if (k == 0) {
            S.vmm.pivot[0] -= shift.x;
            S.vmm.pivot[1] -= shift.y;
            S.vmm.pivot[2] -= shift.z;
          }
        }
        __syncthreads();
        asm_update(S, L, cfg, afterSplit, afterMerge);
        if (threadIdx.x < 32)
          valid = (vmm_is_valid(S.vmm) && suff_is_valid(S.suff) && split_is_valid(S.split)) ? 1u : 0u;
      }
    } else if (fit) {
      valid = 0;
    }
    __syncthreads();
    {
      uint32_t *dst = reinterpret_cast<uint32_t *>(&R.vmm);
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&S.vmm);
      for (int i = threadIdx.x; i < int(sizeof(VMMState) / 4); i += blockDim.x) dst[i] = src[i];
      dst = reinterpret_cast<uint32_t *>(&R.suff);
      src = reinterpret_cast<const uint32_t *>(&S.suff);
      for (int i = threadIdx.x; i < int(sizeof(SuffState) / 4); i += blockDim.x) dst[i] = src[i];
      dst = reinterpret_cast<uint32_t *>(&R.split);
      src = reinterpret_cast<const uint32_t *>(&S.split);
      for (int i = threadIdx.x; i < int(sizeof(SplitState) / 4); i += blockDim.x) dst[i] = src[i];
    }
    if (threadIdx.x == 0) {
      R.afterSplit = afterSplit;
      R.afterMerge = afterMerge;
      R.valid = valid;
      S.report.K = S.vmm.K;
      if (reports) reports[taskId] = S.report;
      if (profiles) {
        S.prof.cycTotal = uint64_t(clock64() - leafStart);
        S.prof.tEnd = global_ns();
        profiles[taskId] = S.prof;
      }
      atomicAdd(finished, 1u);
    }
    __syncthreads();
  }
  // no leaves left: produce for the blocks still working on theirs
  if (!plain) help_others(S, boards, rings, finished, numTasks);
}

PGL_DEFINE_TABLE_UPLOAD(em_upload_tables)

// One thread waits, with the EM kernel's bounded wait, on a flag that nothing
// sets: the wait gives up after limitNs and records its error in *err.
__global__ void bounded_wait_probe_kernel(const uint32_t *flag, int *err, unsigned long long limitNs) {
  if (threadIdx.x == 0 && blockIdx.x == 0) wait_at_least(flag, 1u, err, limitNs);
}
cudaError_t em_bounded_wait_probe(unsigned long long limitNs, int *errOut, cudaStream_t s) {
  uint32_t *flag = nullptr;
  int *err = nullptr;
  cudaError_t e = cudaMalloc(&flag, sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&err, sizeof(int));
  if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, sizeof(uint32_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), s);
  if (e == cudaSuccess) {
    bounded_wait_probe_kernel<<<1, 32, 0, s>>>(flag, err, limitNs);
    count_launch();
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(errOut, err, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (flag) cudaFree(flag);
  if (err) cudaFree(err);
  return e;
}

size_t em_shared_bytes() { return sizeof(EmShared); }

// Shared-pass memory of a launch with `blocks` blocks: the boards, the error
// word and the finished-leaf counter, then one chunk ring per block.
static size_t share_header_bytes(int blocks) {
  return (size_t(blocks) * sizeof(Board) + 2 * sizeof(int) + 255) & ~size_t(255);
}
bool em_tuning_valid(const EmTuning &t) {
  return t.maxHelpers >= 0 && t.maxHelpers <= 64 && t.chunkDiv >= 1 && t.chunkDiv <= 4 && t.stageCap >= 2 &&
         t.stageCap <= kMaxStages && (t.orderByCost == 0 || t.orderByCost == 1) &&
         (t.plainLaunches == 0 || t.plainLaunches == 1) && t.reservedSMs >= 0 && t.reservedSMs < 4096;
}
size_t em_share_bytes(int blocks) { return share_header_bytes(blocks) + size_t(blocks) * kRingFloats * sizeof(float); }
size_t em_share_bytes_plain(int blocks) { return share_header_bytes(blocks); }
size_t em_share_error_offset(int blocks) { return size_t(blocks) * sizeof(Board); }

cudaError_t launch_em(const LeafTask *tasks, uint32_t numTasks, unsigned int *queue, const EmSides &sides,
                      LeafReport *reports, LeafProfile *profiles, void *share, int blocks, const EmTuning &tune,
                      cudaStream_t stream) {
  const size_t smem = sizeof(EmShared);
  // once per process (thread-safe static initialisation)
  static const cudaError_t attr =
      cudaFuncSetAttribute(em_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (attr != cudaSuccess) return attr;
  if (numTasks == 0) return cudaSuccess;
  if (blocks < 1 || share == nullptr || !em_tuning_valid(tune)) return cudaErrorInvalidValue;
  // boards start empty (generation 0, no chunk ready); error word and counter 0
  unsigned char *base = static_cast<unsigned char *>(share);
  cudaError_t e = cudaMemsetAsync(base, 0, share_header_bytes(blocks), stream);
  if (e != cudaSuccess) return e;
  Board *boards = reinterpret_cast<Board *>(base);
  int *err = reinterpret_cast<int *>(base + em_share_error_offset(blocks));
  uint32_t *finished = reinterpret_cast<uint32_t *>(base + em_share_error_offset(blocks) + sizeof(int));
  float *rings = reinterpret_cast<float *>(base + share_header_bytes(blocks));
  // persistent blocks (one per SM: shared memory bound) take leaves from the
  // queue; blocks without a leaf help the others' E-step passes.  The plain
  // form launches one block per region (blocks == numTasks); its blocks use
  // their own boards only, never a chunk ring.
  count_launch();
  em_leaf_kernel<<<unsigned(blocks), kEmThreads, smem, stream>>>(tasks, numTasks, queue, sides, reports, profiles,
                                                                 boards, rings, err, finished, tune);
  return cudaGetLastError();
}

}  // namespace pgl
