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
// accumulator gets the reference's bits.  Scalar per-leaf logic (M step,
// split/merge bookkeeping) runs on thread 0 between passes.
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

enum EmError { kErrNone = 0, kErrChunkWait = 1, kErrSlotWait = 2, kErrCopyWait = 3, kErrLeafTooLarge = 4 };

struct __align__(16) BoardParams {  // one pass as its home block publishes it
  float4 lobeP[3 * kMaxK / 2];
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

struct EmShared {
  VMMState vmm;
  SuffState suff;     // training statistics ("previous" statistics of EM)
  SplitState split;   // training split statistics
  SuffState cur;      // statistics of the current EM iteration
  SuffState temp;     // statistics of a partial refit
  SplitState lsplit;  // split statistics used by the recursive splitting
  Frame invFrame[kMaxK];
  __align__(16) float pbuf[2 * kStageFloats];  // the two pipeline stages
  __align__(16) float4 lobeA[kMaxK + kMaxK / kLanes];  // mean direction, kappa (entry k + k / 8)
  float2 lobeB[kMaxK];                // normalisation, weight
  __align__(16) float4 lobeP[3 * kMaxK / 2];  // E-step passes: two lobes per three entries, see pack_pairs
  __align__(16) float ones[kMaxChunk + 48];  // the factor row of the chains that sum a_k w
  float lobeWInv[kMaxK];              // RN(1 / weight) for div_rcp
  float xch[2][kMaxK];
  uint32_t rcpTab[2048];
  float cost[kMaxK][kMaxK];  // merge cost of components i < j (cost[i][j])
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
  uint32_t validPerWarp[kEmThreads / 32];  // split passes: valid samples per producer warp
  float splitN0[kMaxK];                     // split passes: chi-square counts at the pass start
};
static_assert(offsetof(EmShared, pbuf) % 16 == 0 && offsetof(EmShared, lobeA) % 16 == 0 &&
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
__device__ void vmm_split(VMMState &v, int i0, int i1, float w0, float w1, V3 m0, V3 m1, float mc0, float mc1) {
  v.dist[i1] = v.dist[i0];  // PAVMM.h:225-255
  v.w[i0] = w0; v.mc[i0] = mc0; v.kappa[i0] = mean_cosine_to_kappa(mc0);
  v.mx[i0] = m0.x; v.my[i0] = m0.y; v.mz[i0] = m0.z;
  v.w[i1] = w1; v.mc[i1] = mc1; v.kappa[i1] = mean_cosine_to_kappa(mc1);
  v.mx[i1] = m1.x; v.my[i1] = m1.y; v.mz[i1] = m1.z;
  if (uint32_t(i1) == v.K) v.K++;
  vmm_calc_norm(v);
}
__device__ void vmm_parallax_shift(VMMState &v, V3 s) {  // PAVMM.h:809-831
  int c = vec_count(int(v.K));
  for (int k = 0; k < c * kLanes; ++k) {
    V3 p = mk(v.mx[k], v.my[k], v.mz[k]) * v.dist[k] + s;
    float len = length(p);
    p = p / len;
    bool cond = (v.dist[k] > 0.0f) && (v.dist[k] >= -FLT_MAX) && (v.dist[k] <= FLT_MAX);
    if (cond) { v.mx[k] = p.x; v.my[k] = p.y; v.mz[k] = p.z; }
    v.dist[k] = v.dist[k] > 0.0f ? len : 0.0f;
  }
  v.pivot[0] -= s.x; v.pivot[1] -= s.y; v.pivot[2] -= s.z;
}
__device__ bool vmm_is_valid(const VMMState &v) {  // PAVMM.h:422-513
  bool ok = true;
  for (uint32_t k = 0; k < v.K && k < kMaxK; ++k) {
    ok = ok && isvalidf(v.w[k]) && v.w[k] >= 0.0f && v.w[k] <= 1.0f + 1e-6f;
    ok = ok && isvalidf(v.kappa[k]) && v.kappa[k] >= 0.0f;
    ok = ok && isvalidf(v.mc[k]) && v.mc[k] >= 0.0f && v.mc[k] <= 1.0f;
    ok = ok && isvalidf(v.mx[k]) && v.mx[k] >= -1.0f && v.mx[k] <= 1.0f;
    ok = ok && isvalidf(v.my[k]) && v.my[k] >= -1.0f && v.my[k] <= 1.0f;
    ok = ok && isvalidf(v.mz[k]) && v.mz[k] >= -1.0f && v.mz[k] <= 1.0f;
    ok = ok && isvalidf(v.norm[k]) && v.norm[k] >= 0.0f && isvalidf(v.e2k[k]);
    ok = ok && isvalidf(v.dist[k]) && v.dist[k] >= 0.0f;
  }
  for (uint32_t k = v.K; k < kMaxK; ++k) {
    ok = ok && v.w[k] == 0.0f && v.kappa[k] == 0.0f && v.mx[k] == 0.0f && v.my[k] == 0.0f && v.mz[k] == 1.0f;
    ok = ok && v.mc[k] == 0.0f && fabsf(v.norm[k] - kInv4Pi) < 1e-6f && v.e2k[k] == 1.0f && v.dist[k] == 0.0f;
  }
  return ok;
}

__device__ void suff_clear(SuffState &s, uint32_t K) {
  s.K = K;
  int c = vec_count(int(K));
  for (int k = 0; k < c * kLanes; ++k) s.dx[k] = s.dy[k] = s.dz[k] = s.w[k] = s.dw[k] = 0.0f;
  s.sumWeights = 0.0f; s.numSamples = 0.0f; s.normalized = 0;
}
__device__ void suff_normalize(SuffState &s, float n) {  // WEMFactory.h:553-572
  int c = vec_count(int(s.K));
  s.numSamples = n;
  float sv[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int k = 0; k < c * kLanes; ++k) sv[k % kLanes] += s.w[k];
  s.sumWeights = reduce8(sv);
  float nrm = n / s.sumWeights;
  for (int k = 0; k < c * kLanes; ++k) { s.dx[k] *= nrm; s.dy[k] *= nrm; s.dz[k] *= nrm; s.w[k] *= nrm; }
  s.normalized = 1;
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
__device__ void suff_parallax_shift(SuffState &s, const VMMState &v, V3 shift) {  // WEMFactory.h:265-283
  int c = vec_count(int(v.K));
  for (int k = 0; k < c * kLanes; ++k) {
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
}
__device__ void suff_split(SuffState &s, int i, int j, V3 m0, V3 m1, float mc0, float mc1) {  // WEMFactory.h:516-550
  float sw = s.w[i];
  sw /= 2.0f;
  s.w[i] = sw; s.dx[i] = (m0.x * mc0) * sw; s.dy[i] = (m0.y * mc0) * sw; s.dz[i] = (m0.z * mc0) * sw;
  s.w[j] = sw; s.dx[j] = (m1.x * mc1) * sw; s.dy[j] = (m1.y * mc1) * sw; s.dz[j] = (m1.z * mc1) * sw;
  float t = s.dw[i] * 0.5f;
  s.dw[i] = t; s.dw[j] = t;
  s.K += 1;
}
__device__ void suff_merge(SuffState &s, int i0, int i1) {  // WEMFactory.h:485-513
  int L = int(s.K) - 1;
  s.dx[i0] += s.dx[i1]; s.dy[i0] += s.dy[i1]; s.dz[i0] += s.dz[i1]; s.w[i0] += s.w[i1]; s.dw[i0] += s.dw[i1];
  s.dx[i1] = s.dx[L]; s.dy[i1] = s.dy[L]; s.dz[i1] = s.dz[L]; s.w[i1] = s.w[L]; s.dw[i1] = s.dw[L];
  s.dx[L] = s.dy[L] = s.dz[L] = s.w[L] = s.dw[L] = 0.0f;
  s.K--;
}
__device__ bool suff_is_valid(const SuffState &s) {
  bool ok = true;
  for (uint32_t k = 0; k < s.K && k < kMaxK; ++k)
    ok = ok && isvalidf(s.dx[k]) && isvalidf(s.dy[k]) && isvalidf(s.dz[k]) && isvalidf(s.w[k]) && s.w[k] >= 0.0f &&
         isvalidf(s.dw[k]) && s.dw[k] >= 0.0f;
  for (uint32_t k = s.K; k < kMaxK; ++k)
    ok = ok && s.dx[k] == 0.0f && s.dy[k] == 0.0f && s.dz[k] == 0.0f && s.w[k] == 0.0f && s.dw[k] == 0.0f;
  return ok && isvalidf(s.numSamples) && s.numSamples >= 0.0f && isvalidf(s.sumWeights) && s.sumWeights >= 0.0f;
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
  bool lane[kLanes];
  for (int j = 0; j < kLanes; ++j) lane[j] = true;
  for (int k = 0; k < kMaxK; ++k) {
    bool ok = isvalidf(s.mx[k]) && isvalidf(s.my[k]) && isvalidf(s.cx[k]) && isvalidf(s.cy[k]) && isvalidf(s.cz[k]) &&
              isvalidf(s.chi2[k]) && s.chi2[k] >= 0.0f && isvalidf(s.sw[k]) && s.sw[k] >= 0.0f && isvalidf(s.sa[k]) &&
              s.sa[k] >= 0.0f && isvalidf(s.n[k]) && s.n[k] >= 0.0f;
    lane[k % kLanes] = lane[k % kLanes] && ok;
  }
  bool any = false;
  for (int j = 0; j < kLanes; ++j) any = any || lane[j];
  return any && s.K > 0 && s.K <= kMaxK;
}

// MAP M-step (WEMFactory.h:895-1148); mask == nullptr is the full step.
__device__ void map_step(VMMState &v, const SuffState &cur, const SuffState &prev, const FieldConfig &cfg, const int *mask) {
  int c = vec_count(int(v.K));
  float K = float(v.K);
  float N = cur.numSamples + prev.numSamples;
  int rem = int(v.K % kLanes);
  if (!mask) {
    for (int k = 0; k < c * kLanes; ++k) {
      float w = cur.w[k] + prev.w[k];
      v.w[k] = (cfg.weightPrior + w) / ((cfg.weightPrior * K) + N);
    }
  } else {
    float sw[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0}, sp[kLanes] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int k = 0; k < c * kLanes; ++k) {
      float w = cur.w[k] + prev.w[k];
      w = (cfg.weightPrior + w) / ((cfg.weightPrior * K) + N);
      sp[k % kLanes] += mask[k] ? w : 0.0f;
      sw[k % kLanes] += mask[k] ? 0.0f : v.w[k];
      v.w[k] = mask[k] ? w : v.w[k];
    }
    float inv = 1.0f / reduce8(sp);
    inv *= 1.0f - reduce8(sw);
    for (int k = 0; k < c * kLanes; ++k) v.w[k] = mask[k] ? v.w[k] * inv : v.w[k];
  }
  if (rem > 0)
    for (int i = rem; i < kLanes; ++i) v.w[(c - 1) * kLanes + i] = 0.0f;

  float curN = cur.numSamples, prevN = prev.numSamples, NN = curN + prevN;
  float overallN = cur.numSamples + prev.overallNumSamples;
  float curW = curN / NN, prevW = 1.0f - curW;
  for (int k = 0; k < c * kLanes; ++k) {
    float partialN = v.w[k] * overallN;
    V3 cm = cur.w[k] > 0.0f ? mk(cur.dx[k] / cur.w[k], cur.dy[k] / cur.w[k], cur.dz[k] / cur.w[k]) : mk(0, 0, 0);
    V3 pm = prev.w[k] > 0.0f ? mk(prev.dx[k] / prev.w[k], prev.dy[k] / prev.w[k], prev.dz[k] / prev.w[k]) : mk(0, 0, 0);
    V3 md = cm * curW + pm * prevW;
    float mc = length(md);
    bool upd = mask ? (mask[k] != 0) : true;
    if (upd && mc > 0.0f) { v.mx[k] = md.x / mc; v.my[k] = md.y / mc; v.mz[k] = md.z / mc; }
    mc = (cfg.mcPrior * cfg.mcPriorStrength + mc * partialN) / (cfg.mcPriorStrength + partialN);
    mc = emin(cfg.maxMeanCosine, mc);
    if (upd) { v.mc[k] = mc; v.kappa[k] = mean_cosine_to_kappa(mc); }
  }
  if (rem > 0)
    for (int i = rem; i < kLanes; ++i) {
      int k = (c - 1) * kLanes + i;
      v.mx[k] = 0.0f; v.my[k] = 0.0f; v.mz[k] = 1.0f; v.mc[k] = 0.0f; v.kappa[k] = 0.0f;
      if (!mask) { v.norm[k] = kInv4Pi; v.e2k[k] = 1.0f; }
    }
  vmm_calc_norm(v);
}

// suff_normalize and map_step by one warp, lane k doing lobe k: every lobe's
// arithmetic is the scalar functions' own; the sums over lobes keep the
// scalar order (vfloat8 lane sums over k, then the 8-lane reduction) on lane 0.
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

// SplitComponent (Splitter.h:527-665)
__device__ bool split_component(VMMState &v, SplitState &sp, SuffState &suff, int idx, const FieldConfig &cfg) {
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
  float nw0 = w * 0.5f, nw1 = nw0;
  V3 m0 = mu, m1 = mu;
  float nmc0 = mc, nmc1 = mc * mc;
  if (D > 1e-8f) {
    float ax = (e0x * ev0) * 0.5f, ay = (e0y * ev0) * 0.5f;
    Frame fr = frame_of(mu, false);
    m0 = xfm(fr, map2d_to_3d(meanx + ax, meany + ay));
    nmc0 = mc / fabsf(dot(mu, m0));
    nmc0 = smin(nmc0, cfg.maxMeanCosineSplit);
    nmc1 = nmc0;
    m1 = xfm(fr, map2d_to_3d(meanx - ax, meany - ay));
  } else {
    if (numAssigned < 2.0f) return false;
  }
  int K = int(v.K);
  vmm_split(v, idx, K, nw0, nw1, m0, m1, nmc0, nmc1);
  suff_split(suff, idx, K, m0, m1, nmc0, nmc1);
  split_zero_lane(sp, idx);
  split_zero_lane(sp, K);
  sp.K = uint32_t(K + 1);
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
__device__ float merge_cost(const VMMState &v, int i0, int i1) {  // Merger.h:92-177
  float w0 = v.w[i0], k0 = v.kappa[i0], mc0 = v.mc[i0], n0 = v.norm[i0];
  float w1 = v.w[i1], k1 = v.kappa[i1], mc1 = v.mc[i1], n1 = v.norm[i1];
  V3 m0 = mk(v.mx[i0], v.my[i0], v.mz[i0]), m1 = mk(v.mx[i1], v.my[i1], v.mz[i1]);
  if (i0 == i1) { w0 /= 2.0f; w1 /= 2.0f; }
  float w = w0 + w1, kappa = 0.0f, nrm = kInv4Pi, e2k = 1.0f;
  V3 m = m0 * (w0 * mc0) + m1 * (w1 * mc1);
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
  V3 nm = mk(-m.x, -m.y, -m.z);
  V3 m00, m11, m01;
  float k00, k11, k01, n00, n11, n01;
  float s00 = product_scale(m0, k0, n0, m0, k0, n0, m00, k00, n00);
  float s11 = product_scale(m1, k1, n1, m1, k1, n1, m11, k11, n11);
  float s01 = product_scale(m0, k0, n0, m1, k1, n1, m01, k01, n01);
  float w00 = w0 * w0, w11 = w1 * w1, w01 = w0 * w1;
  float chi = 0.0f;
  chi += (w00 / w) * (s00 * integrated_division(m00, k00, n00, nm, kappa, nrm, e2k));
  chi += (w11 / w) * (s11 * integrated_division(m11, k11, n11, nm, kappa, nrm, e2k));
  chi += 2.0f * (w01 / w) * (s01 * integrated_division(m01, k01, n01, nm, kappa, nrm, e2k));
  chi -= w;
  return chi;
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
// shared-memory stages:
//   producers (threads [0, C * parts)): `parts` adjacent lanes per sample, one
//     SIMD vector of 8 lobes each; the lobe terms in registers, the sample pdf
//     (vfloat8 lane sums carried from part to part in lobe-vector order, then
//     the 8-lane reduction), then the finished term of every accumulator for
//     their lobes written to stage (c & 1);
//   consumers (threads [P, 512)): one thread per accumulator (for example the
//     x component of lobe 7's weighted direction sum), adding the chunk in
//     stage ((c - 1) & 1) in sample order.
// The consumers keep the reference's summation order (sequential over samples
// within each SIMD lane).  Samples that the reference skips (pdf <= 1e-16)
// contribute a term of exactly +-0, which leaves an accumulator unchanged:
// accumulators start at +0 and a round-to-nearest sum that starts at +0 never
// becomes -0.  Consumer lanes only load and add, so chain warps do not diverge
// (chi-square lanes have a warp of their own).  Each pass gives the consumers
// the warps its chains need and the producers the rest; the chunk size
// follows from the stage memory and the producer threads.  E-step passes
// (most of the work) use the same roles, with a loader warp besides, and can
// take chunks made by other blocks (below).

struct LeafSamples {
  const float4 *dirw;  // direction xyz, weight
  const float *pdf;
  const float *dist;
  uint32_t count;
};

enum PassKind { kPassDistance = 1, kPassSplit = 2 };  // in-block passes

// Thread roles and stage layout of one pass (the same in every thread).
struct PassShape {
  int P;        // threads [P, kEmThreads) consume
  int parts;    // producer lanes per sample (lobe vectors, 3 rounded to 4)
  int C;        // samples per chunk
  int threads;  // producer threads: C * parts, a multiple of 32
  int R;        // row stride of the per-(lobe, sample) rows: C + 2 floats
  int stage;    // floats per stage
};
template <PassKind kind>
__device__ __forceinline__ PassShape pass_shape(int Kp, int budget = kStageFloats) {
  // rows: one per (accumulator, lobe); extra: per-sample arrays
  int consWarps, rows, extra;
  if (kind == kPassDistance) {  // 2 Kp chains
    consWarps = (2 * Kp + 31) / 32;
    rows = 2 * Kp;
    extra = 0;
  } else {  // 5 Kp product chains, two per lane, then (from a warp boundary) Kp chi-square chains
    consWarps = (5 * Kp + 63) / 64 + 1;
    rows = 7 * Kp;  // a, a w, three covariance terms, chi, 1/n
    extra = 1;      // validity
  }
  PassShape p;
  const int cnt = Kp / kLanes;
  p.parts = cnt == 3 ? 4 : cnt;
  p.P = kEmThreads - 32 * consWarps;
  int c = (budget - 2 * rows) / (rows + extra);
  const int byThreads = p.P / p.parts;
  c = c < byThreads ? c : byThreads;
  // C * parts a multiple of 32 (whole warps) and C a multiple of 8.  Rows of
  // C + 2 floats: (C + 2) / 2 is odd, so the consumers' 64-bit loads of
  // consecutive rows fall in distinct banks, and rows 8 apart are 16 banks
  // apart, so two parts of a sample store to distinct banks.
  const int mult = 32 / p.parts > 8 ? 32 / p.parts : 8;
  p.C = c - c % mult;
  p.threads = p.C * p.parts;
  p.R = p.C + 2;
  p.stage = rows * p.R + extra * p.C;
  return p;
}

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

// Lobe parameters packed for the producers' broadcast loads.
__device__ void pack_lobes(EmShared &S, int Kp) {
  const int tid = threadIdx.x;
  if (tid < Kp) {
    const VMMState &v = S.vmm;
    // entry k + k / 8: the parts of a sample read lobes k and k + 8 at once
    S.lobeA[tid + (tid >> 3)] = make_float4(v.mx[tid], v.my[tid], v.mz[tid], v.kappa[tid]);
    S.lobeB[tid] = make_float2(v.norm[tid], v.w[tid]);
    S.lobeWInv[tid] = rcp_for_div(v.w[tid]);
  }
}

// The lobe parameters of an E-step pass by pairs of lobes, for packed
// arithmetic: {x0, x1, y0, y1}, {z0, z1, kappa0, kappa1}, {norm0, norm1, w0, w1}.
__device__ void pack_pairs(EmShared &S, int Kp) {
  const int i = int(threadIdx.x);
  if (2 * i < Kp) {
    const VMMState &v = S.vmm;
    const int k = 2 * i;
    S.lobeP[3 * i] = make_float4(v.mx[k], v.mx[k + 1], v.my[k], v.my[k + 1]);
    S.lobeP[3 * i + 1] = make_float4(v.mz[k], v.mz[k + 1], v.kappa[k], v.kappa[k + 1]);
    S.lobeP[3 * i + 2] = make_float4(v.norm[k], v.norm[k + 1], v.w[k], v.w[k + 1]);
  }
}

// One producer lane's view of a sample: the E-step terms of its 8 lobes
// (vector v), then the sample pdf and 1/pdf shared by all parts.
struct PartTerms {
  float t[kLanes];
  float pdf, inv;
  bool valid;
};
__device__ __forceinline__ void part_terms(const EmShared &S, int cnt, int parts, int v, bool have, V3 d,
                                           PartTerms &T) {
  const unsigned full = 0xFFFFFFFFu;
  if (have && v < cnt) {
#pragma unroll
    for (int j = 0; j < kLanes; ++j) {
      const int k = v * kLanes + j;
      const float4 A = S.lobeA[k + v];
      const float2 B = S.lobeB[k];
      float ct = dot(d, mk(A.x, A.y, A.z));
      float cm1 = emin(ct - 1.0f, 0.0f);
      float ev = B.x * fexp(A.w * cm1);
      T.t[j] = B.y * ev;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kLanes; ++j) T.t[j] = 0.0f;
  }
  // lane sums over the lobe vectors in order: ((t0 + t1) + t2) + t3
  float p[kLanes];
#pragma unroll
  for (int j = 0; j < kLanes; ++j) p[j] = T.t[j];
  for (int step = 1; step < parts; ++step) {
#pragma unroll
    for (int j = 0; j < kLanes; ++j) {
      const float in = __shfl_up_sync(full, p[j], 1);
      if (v == step) p[j] = in + T.t[j];
    }
  }
  float pdf = 0.0f, inv = 0.0f;
  bool valid = false;
  if (v == parts - 1 && have) {
    pdf = reduce8(p);
    valid = pdf > 1e-16f;
    inv = valid ? rcp_avx2_tab(pdf, S.rcpTab) : 0.0f;
  }
  const int last = (int(threadIdx.x & 31) - v) + parts - 1;
  T.pdf = __shfl_sync(full, pdf, last);
  T.inv = __shfl_sync(full, inv, last);
  T.valid = __shfl_sync(full, valid ? 1 : 0, last) != 0;
}

struct SampleIn {
  float4 dw;
  float x;  // pdf (split pass) or distance (distance pass)
  bool have;
};
template <PassKind kind>
__device__ __forceinline__ SampleIn load_sample(const LeafSamples &L, uint32_t idx) {
  SampleIn r;
  r.have = idx < L.count;
  r.dw = make_float4(0.f, 0.f, 0.f, 0.f);
  r.x = 0.0f;
  if (r.have) {
    r.dw = L.dirw[idx];
    if constexpr (kind == kPassDistance) r.x = L.dist[idx];
    else if constexpr (kind == kPassSplit) r.x = L.pdf[idx];
  }
  return r;
}

// a / b in a function of its own: the rare operands that div_rcp_try leaves
// over.  As a plain expression behind a condition the division is evaluated
// for every operand and the result selected afterwards; its slow path for
// small numerators (most lobes are far from a sample's direction) was then
// half of a split-statistics pass, and a branch per quotient keeps the eight
// lobes of a lane from overlapping.  So a lane does its lobes without a
// branch and then once more those that need it (first Update with 1,048,576
// samples: split passes 182 -> 105 cycles per sample, distance passes 19 ->
// 16, the Update 17.7 -> 11.7 ms).
__device__ __noinline__ float div_plain(float a, float b) { return a / b; }

// Producer: lane v of sample slot s fills its lobes' rows of stage B.  In
// split passes the running count of valid samples (for the chi-square means'
// 1/n) needs a prefix over the chunk: warp ballots, then a barrier among the
// producer threads only (named barrier 1), then `base` (valid samples of the
// earlier chunks) moves on by the chunk's total.
template <PassKind kind>
__device__ __forceinline__ void produce(EmShared &S, const PassShape &sh, int cnt, int Kp, int s, int v,
                                        const SampleIn &in, float *B, uint32_t &base) {
  PartTerms T;
  const V3 d = mk(in.dw.x, in.dw.y, in.dw.z);
  const float w = in.dw.w;
  part_terms(S, cnt, sh.parts, v, in.have, d, T);
  const bool valid = in.have && T.valid;
  const int R = sh.R;
  const bool mine = v < cnt;  // this lane has lobes
  if constexpr (kind == kPassDistance) {
    // rows k: wts * rcp(distance); rows Kp + k: wts
    if (mine) {
      const float sd = valid ? rcp_avx2_tab(in.x, S.rcpTab) : 0.0f;
      unsigned redo = 0;  // lobes whose quotient div_rcp_try could not give
#pragma unroll
      for (int j = 0; j < kLanes; ++j) {
        const int k = v * kLanes + j;
        bool ok = true;
        const float a = T.t[j] * T.inv;
        float wts = (w * a) * div_rcp_try(a * T.pdf, S.lobeB[k].y, S.lobeWInv[k], ok);
        if (!valid) wts = 0.0f;
        redo |= ok ? 0u : 1u << j;
        B[k * R + s] = wts * sd;
        B[(Kp + k) * R + s] = wts;
      }
      if (valid && redo != 0) {
#pragma unroll
        for (int j = 0; j < kLanes; ++j) {
          if ((redo >> j & 1u) == 0) continue;
          const int k = v * kLanes + j;
          const float a = T.t[j] * T.inv;
          const float wts = (w * a) * div_plain(a * T.pdf, S.lobeB[k].y);
          B[k * R + s] = wts * sd;
          B[(Kp + k) * R + s] = wts;
        }
      }
    }
  } else {
    // count of valid samples up to and including this one
    const unsigned full = 0xFFFFFFFFu;
    const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
    const unsigned b = __ballot_sync(full, v == 0 && valid);
    if (lane == 0) S.validPerWarp[warp] = uint32_t(__popc(b));
    asm volatile("bar.sync 1, %0;" ::"r"(sh.threads) : "memory");
    uint32_t before = 0, total = 0;
    for (int q = 0; q < sh.threads / 32; ++q) {
      const uint32_t n = S.validPerWarp[q];
      before += q < warp ? n : 0u;
      total += n;
    }
    const uint32_t count = base + before + uint32_t(__popc(b & ((1u << (lane - v)) - 1u))) + 1u;
    base += total;
    // rows r Kp + k: a, a w, (a w)(lx lx), (a w)(ly ly), (a w)(lx ly), chi,
    // RN(1 / n) with n = n0_k + count; then the validity per sample
    const float spdfv = in.x;
    const float value = w * spdfv;
    const float mcEst = S.mcEstimate;
    // the three divisors are per sample: one reciprocal each, then Markstein
    const float den1 = mcEst * T.pdf, den2 = ((mcEst * mcEst) * T.pdf) * T.pdf;
    const float y1 = rcp_for_div(den1), y2 = rcp_for_div(den2), y3 = rcp_for_div(spdfv);
    if (mine) {
      const float vv = value * value;
      unsigned redo = 0;  // lobes with a quotient that div_rcp_try could not give
#pragma unroll
      for (int j = 0; j < kLanes; ++j) {
        const int k = v * kLanes + j;
        bool ok = true;
        const float a = valid ? T.t[j] * T.inv : 0.0f;
        const float vmf = a * T.pdf;
        const float pvp = div_rcp_try(vmf * value, den1, y1, ok);
        float chi = div_rcp_try(vv * vmf, den2, y2, ok);
        chi -= 2.0f * pvp;
        chi += vmf;
        chi = div_rcp_try(chi, spdfv, y3, ok);
        chi = a > 0.0f ? chi : 0.0f;
        redo |= ok | !valid ? 0u : 1u << j;
        const V3 ld = xfm(S.invFrame[k], d);
        const float aw = a * w;
        const float n = S.splitN0[k] + float(count);
        B[k * R + s] = a;
        B[(Kp + k) * R + s] = valid ? aw : 0.0f;
        B[(2 * Kp + k) * R + s] = valid ? aw * (ld.x * ld.x) : 0.0f;
        B[(3 * Kp + k) * R + s] = valid ? aw * (ld.y * ld.y) : 0.0f;
        B[(4 * Kp + k) * R + s] = valid ? aw * (ld.x * ld.y) : 0.0f;
        B[(5 * Kp + k) * R + s] = valid ? chi : 0.0f;
        B[(6 * Kp + k) * R + s] = (valid & (n >= 1e-30f) & (n <= 1e30f)) ? rcp_rn(n) : 0.0f;
      }
      if (redo != 0) {
#pragma unroll
        for (int j = 0; j < kLanes; ++j) {
          if ((redo >> j & 1u) == 0) continue;
          const float a = T.t[j] * T.inv;
          const float vmf = a * T.pdf;
          const float pvp = div_plain(vmf * value, den1);
          float chi = div_plain(vv * vmf, den2);
          chi -= 2.0f * pvp;
          chi += vmf;
          chi = div_plain(chi, spdfv);
          B[(5 * Kp + v * kLanes + j) * R + s] = a > 0.0f ? chi : 0.0f;
        }
      }
    }
    if (v == 0) B[7 * Kp * R + s] = valid ? 1.0f : 0.0f;
  }
}

__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ float4 ld4(const float *p) {  // two 64-bit loads (rows are 8-byte aligned)
  const float2 a = ld2(p), b = ld2(p + 2);
  return make_float4(a.x, a.y, b.x, b.y);
}

// Sum of one row (the terms of one accumulator) in sample order; loads run 8
// samples ahead of the additions.
__device__ __forceinline__ void row_chain(const float *row, int n4, float &acc) {
  int s = 0;
  if (n4 >= 8) {
    float4 a = ld4(row), b = ld4(row + 4);
    for (; s + 8 <= n4; s += 8) {
      const int sn = s + 16 <= n4 ? s + 8 : s;
      const float4 a1 = ld4(row + sn), b1 = ld4(row + sn + 4);
      acc += a.x;
      acc += a.y;
      acc += a.z;
      acc += a.w;
      acc += b.x;
      acc += b.y;
      acc += b.z;
      acc += b.w;
      a = a1;
      b = b1;
    }
  }
  if (s < n4) {
    const float4 v = ld4(row + s);
    acc += v.x;
    acc += v.y;
    acc += v.z;
    acc += v.w;
  }
}

// Distance pass (WEMFactory.h:1199-1326): lanes c < Kp sum wts * rcp(distance),
// lanes Kp <= c < 2 Kp sum wts.
__device__ __forceinline__ void distance_chain(const float *B, const PassShape &sh, int c, int Kp, int n4,
                                               float &acc) {
  if (c < 2 * Kp) row_chain(B + c * sh.R, n4, acc);
}

// Split-statistics pass (Splitter.h:439-523).  Lanes c < 5 Kp sum row c
// (r = c / Kp: sumAssignedSamples a, sumWeights a w, then the 2D covariance
// sums (a w)(lx lx), (a w)(ly ly), (a w)(lx ly)).  Chi-square lanes start at
// the next warp: the running mean chi2 += (chi - chi2) / n over the valid
// samples, n counting from n0.  Markstein's steps with the producers'
// y = RN(1 / (n0 + count)) give (chi - chi2) / n exactly (a skipped sample,
// y = 0, adds +-0) when y belongs to the lane's own running count n (the
// usual case: n equals n0 + count) and the difference d and the quotient lie
// in [1e-30, 1e30] (or d is 0).  The chain checks this per group of four
// samples beside the additions, not between them: the counts, the largest
// |d| against 1e30 and the smallest non-zero |d| against 1e-30 times the
// group's last n (so every quotient of the group is in range).  From the
// first group that fails (rare) the chunk is summed again with divisions,
// which give the same bits wherever Markstein's steps were exact.
__device__ __forceinline__ int split_chi_base(int Kp) { return ((5 * Kp + 63) / 64) * 32; }
__device__ __forceinline__ void split_chain(const float *B, const PassShape &sh, int c, int Kp, int n4, float n0,
                                            float &acc, float &acc2, float &accN, float &cnt) {
  const int R = sh.R;
  const int chiBase = split_chi_base(Kp);
  if (c < chiBase) {  // rows c and c + chiBase (a row chain costs a few cycles per sample, the chi chain ~50)
    if (c < 5 * Kp) row_chain(B + c * R, n4, acc);
    if (c + chiBase < 5 * Kp) row_chain(B + (c + chiBase) * R, n4, acc2);
  } else if (c < chiBase + Kp) {
    const int k = c - chiBase;
    const float *xr = B + (5 * Kp + k) * R, *yr = B + (6 * Kp + k) * R, *vr = B + 7 * Kp * R;
    const float accStart = acc, nStart = accN;
    int redoAt = n4;  // first group that failed the range check
    float accRedo = 0.0f, nRedo = 0.0f;
    float4 x = ld4(xr), y = ld4(yr), v = ld4(vr);
    for (int s = 0; s < n4; s += 4) {
      const int sn = s + 4 < n4 ? s + 4 : s;
      const float4 x1 = ld4(xr + sn), y1 = ld4(yr + sn), v1 = ld4(vr + sn);
      const float accG = acc, nG = accN;
      const float n1 = accN + v.x, n2 = n1 + v.y, n3 = n2 + v.z, n4v = n3 + v.w;
      const float c1 = cnt + v.x, c2 = c1 + v.y, c3 = c2 + v.z, c4 = c3 + v.w;
      const bool same = (v.x == 0.0f || n1 == n0 + c1) & (v.y == 0.0f || n2 == n0 + c2) &
                        (v.z == 0.0f || n3 == n0 + c3) & (v.w == 0.0f || n4v == n0 + c4);
      const float d1 = x.x - acc;
      acc = acc + markstein_q(d1, n1, y.x);
      const float d2 = x.y - acc;
      acc = acc + markstein_q(d2, n2, y.y);
      const float d3 = x.z - acc;
      acc = acc + markstein_q(d3, n3, y.z);
      const float d4 = x.w - acc;
      acc = acc + markstein_q(d4, n4v, y.w);
      const float a1 = fabsf(d1), a2 = fabsf(d2), a3 = fabsf(d3), a4 = fabsf(d4);
      const float gMax = fmaxf(fmaxf(a1, a2), fmaxf(a3, a4));
      const float gMin = fminf(fminf(a1 == 0.0f ? INFINITY : a1, a2 == 0.0f ? INFINITY : a2),
                               fminf(a3 == 0.0f ? INFINITY : a3, a4 == 0.0f ? INFINITY : a4));
      if ((!same || !(gMax <= 1e30f) || gMin < 1.0000002e-30f * n4v) && redoAt == n4) {
        redoAt = s;
        accRedo = accG;
        nRedo = nG;
      }
      accN = n4v;
      cnt = c4;
      x = x1;
      y = y1;
      v = v1;
    }
    if (acc != acc) {
      redoAt = 0;
      accRedo = accStart;
      nRedo = nStart;
    }
    if (redoAt < n4) {
      acc = accRedo;
      accN = nRedo;
      for (int s = redoAt; s < n4; ++s) {
        const float vv = vr[s];
        accN += vv;
        if (vv != 0.0f) acc += (xr[s] - acc) / accN;
      }
    }
  }
}

// Runs one distance or split-statistics pass over the leaf's samples in the
// home block.  `acc`/`accN` are the consumer's accumulators (initialised by
// the caller); chunk c is made into stage (c & 1) while the consumers add
// chunk c - 1.
template <PassKind kind>
__device__ __noinline__ void run_pass(EmShared &S, const LeafSamples &L, const PassShape &sh, int cnt, float &accOut,
                                      float &acc2Out, float &accNOut) {
  const int tid = threadIdx.x;
  float acc = accOut, acc2 = acc2Out, accN = accNOut;  // the chains run on registers
  const int Kp = cnt * kLanes;
  const int C = sh.C;
  const uint32_t rounds = (L.count + C - 1) / C;
  const bool producer = tid < sh.threads;
  const int s = tid / sh.parts, v = tid % sh.parts;
  const bool consumer = tid >= sh.P;
  const int c = tid - sh.P;
  const int chiK = kind == kPassSplit ? c - split_chi_base(Kp) : -1;
  const float n0 = (chiK >= 0 && chiK < Kp) ? S.splitN0[chiK] : 0.0f;
  float count = 0.0f;
  uint32_t base = 0;
  SampleIn next;
  if (producer) next = load_sample<kind>(L, uint32_t(s));
  long long cycP = 0, cycC = 0;
  for (uint32_t it = 0; it <= rounds; ++it) {
    if (producer && it < rounds) {
      const long long t0 = clock64();
      const SampleIn cur = next;
      if (it + 1 < rounds) next = load_sample<kind>(L, (it + 1) * C + s);
      produce<kind>(S, sh, cnt, Kp, s, v, cur, S.pbuf + (it & 1) * kStageFloats, base);
      cycP += clock64() - t0;
    }
    if (consumer && it >= 1) {
      const long long t0 = clock64();
      const uint32_t chunk = it - 1;
      const int n = int(min(uint32_t(C), L.count - chunk * C));
      const int n4 = (n + 3) & ~3;
      const float *B = S.pbuf + (chunk & 1) * kStageFloats;
      if constexpr (kind == kPassDistance) distance_chain(B, sh, c, Kp, n4, acc);
      else split_chain(B, sh, c, Kp, n4, n0, acc, acc2, accN, count);
      cycC += clock64() - t0;
    }
    __syncthreads();
  }
  accOut = acc;
  acc2Out = acc2;
  accNOut = accN;
  const int probe = kind == kPassSplit ? split_chi_base(Kp) : 0;
  if (tid == 0 && kind == kPassSplit) S.prof.cycProdS += uint64_t(cycP);
  if (c == probe && kind == kPassSplit) S.prof.cycConsS += uint64_t(cycC);
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
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }
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

// Two lobes' E-step terms w norm fexp(kappa min(cos - 1, 0)) of direction d.
// The multiplications are packed (each component rounds as its own multiply),
// the additions are not: the compiler contracts a packed multiply and a packed
// addition into one rounding.  The exponential's argument is not positive (or NaN):
// below -100 the result is 0 either way, so the argument is clamped there
// (NaN kept) and the scale's exponent clamped at 0; the rest is fexp's.
__device__ __forceinline__ float2 pair_terms(float4 xy, float4 zk, float4 nw, V3 d) {
  const float ln2Part1 = float(0.6931457519), ln2Part2 = float(1.4286067653e-6);
  float2 c = __fmul2_rn(make_float2(d.z, d.z), make_float2(zk.x, zk.y));
  c = __ffma2_rn(make_float2(d.y, d.y), make_float2(xy.z, xy.w), c);
  c = __ffma2_rn(make_float2(d.x, d.x), make_float2(xy.x, xy.y), c);
  // fminf(NaN, 0) is 0, as the reference's MINPS
  float2 v = __fmul2_rn(make_float2(zk.z, zk.w), make_float2(fminf(c.x - 1.0f, 0.0f), fminf(c.y - 1.0f, 0.0f)));
  asm("max.NaN.f32 %0, %0, 0fC2C80000;" : "+f"(v.x));  // -100
  asm("max.NaN.f32 %0, %0, 0fC2C80000;" : "+f"(v.y));
  const float2 sc = __fmul2_rn(v, make_float2(1.44269502162933349609375f, 1.44269502162933349609375f));
  const float t0 = __fadd_rd(sc.x, 12582912.0f), t1 = __fadd_rd(sc.y, 12582912.0f);  // floor, see fexp
  const float2 kr = make_float2(t0 - 12582912.0f, t1 - 12582912.0f);
  const uint32_t e0 = uint32_t(max(int(f2u(t0)) - (0x4B400000 - 127), 0)) << 23;
  const uint32_t e1 = uint32_t(max(int(f2u(t1)) - (0x4B400000 - 127), 0)) << 23;
  float2 m = __fmul2_rn(kr, make_float2(ln2Part1, ln2Part1));
  float2 x = make_float2(v.x - m.x, v.y - m.y);
  m = __fmul2_rn(kr, make_float2(ln2Part2, ln2Part2));
  x = make_float2(x.x - m.x, x.y - m.y);
  float2 r = __fmul2_rn(x, make_float2(2.7555381529964506626129150390625e-4f, 2.7555381529964506626129150390625e-4f));
  const float coeff[7] = {1.304379315115511417388916015625e-3f, 8.378830738365650177001953125e-3f,
                          4.16539050638675689697265625e-2f, 0.166668415069580078125f,
                          0.4999999105930328369140625f, 1.0f, 1.0f};
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    r = make_float2(r.x + coeff[i], r.y + coeff[i]);
    r = i < 6 ? __fmul2_rn(x, r) : __fmul2_rn(r, make_float2(u2f(e0), u2f(e1)));
  }
  return __fmul2_rn(make_float2(nw.z, nw.w), __fmul2_rn(make_float2(nw.x, nw.y), r));
}

// Producers: `nthreads` threads (index t) fill chunk `chunk` into G (a stage
// or a ring slot), a sample per thread with the terms of all its lobes in
// registers: the lobe vectors' sums stay in order without shuffles, the 32
// lobes give independent work to cover the exponentials' latency, the lobe
// parameters are broadcast loads and a warp stores whole rows.  Issue bound:
// 30 FP32 operations and about as many issue slots per lobe, 15 cycles per
// sample at 32 lobes alone on an SM.  A lane per lobe vector and sample, with
// shuffles between the vectors, held a leaf of 30 lobes that no other block
// helps at 39 cycles per sample and pass; it now takes 28.
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
        term[i] = pair_terms(S.lobeP[3 * i], S.lobeP[3 * i + 1], S.lobeP[3 * i + 2], d);
        p[j] = v == 0 ? term[i] : make_float2(p[j].x + term[i].x, p[j].y + term[i].y);
      }
    const float pdf = ((p[0].x + p[0].y) + (p[1].x + p[1].y)) + ((p[2].x + p[2].y) + (p[3].x + p[3].y));  // reduce8
    const bool valid = have && pdf > 1e-16f;
    const float inv = valid ? rcp_avx2_tab(pdf, S.rcpTab) : 0.0f;
    float *row = G + s;
#pragma unroll
    for (int i = 0; i < Kp / 2; ++i) {
      const float2 a = __fmul2_rn(term[i], make_float2(inv, inv));
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
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void add4(float &acc, float4 v) {
  acc += v.x;
  acc += v.y;
  acc += v.z;
  acc += v.w;
}
__device__ __forceinline__ float4 chain_terms(float4 a, float4 d, float4 w) {
  const float2 p0 = __fmul2_rn(__fmul2_rn(make_float2(d.x, d.y), make_float2(a.x, a.y)), make_float2(w.x, w.y));
  const float2 p1 = __fmul2_rn(__fmul2_rn(make_float2(d.z, d.w), make_float2(a.z, a.w)), make_float2(w.z, w.w));
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
    for (int i = 0; i < 3 * Kp / 2; ++i) bp.lobeP[i] = S.lobeP[i];
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
        for (int i = tid; i < 3 * kMaxK / 2; i += kEmThreads) S.lobeP[i] = __ldcg(&src.lobeP[i]);
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
  const PassShape sh = pass_shape<kPassDistance>(Kp);
  pack_lobes(S, Kp);
  __syncthreads();
  float acc = 0.0f, accN = 0.0f;
  float unused = 0.0f;
  run_pass<kPassDistance>(S, L, sh, cnt, acc, unused, accN);
  // exchange: bd in xch[0][k], bw in xch[1][k]
  const int c = tid - sh.P;
  if (c >= 0 && c < 2 * Kp) S.xch[c / Kp][c % Kp] = acc;
  __syncthreads();
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
  const PassShape sh = pass_shape<kPassSplit>(Kp);
  if (tid < Kp) {
    S.invFrame[tid] = inverse_of(frame_of(mk(S.vmm.mx[tid], S.vmm.my[tid], S.vmm.mz[tid]), true));
    S.splitN0[tid] = sp.n[tid];
  }
  pack_lobes(S, Kp);
  __syncthreads();
  const int c = tid - sh.P;
  const int chiBase = split_chi_base(Kp);
  // row q < 5 Kp: r = q / Kp selects sa, sw, cx, cy, cz of lobe k = q % Kp
  auto row_value = [&](int q) {
    const int r = q / Kp, k = q % Kp;
    return r == 0 ? sp.sa[k] : r == 1 ? sp.sw[k] : r == 2 ? sp.cx[k] : r == 3 ? sp.cy[k] : sp.cz[k];
  };
  auto row_store = [&](int q, float v) {
    const int r = q / Kp, k = q % Kp;
    if (r == 0) sp.sa[k] = v;
    else if (r == 1) sp.sw[k] = v;
    else if (r == 2) sp.cx[k] = v;
    else if (r == 3) sp.cy[k] = v;
    else sp.cz[k] = v;
  };
  float acc = 0.0f, acc2 = 0.0f, accN = 0.0f;
  if (c >= 0 && c < chiBase) {
    if (c < 5 * Kp) acc = row_value(c);
    if (c + chiBase < 5 * Kp) acc2 = row_value(c + chiBase);
  } else if (c >= chiBase && c < chiBase + Kp) {
    acc = sp.chi2[c - chiBase];
    accN = sp.n[c - chiBase];
  }
  run_pass<kPassSplit>(S, L, sh, cnt, acc, acc2, accN);
  if (c >= 0 && c < chiBase) {
    if (c < 5 * Kp) row_store(c, acc);
    if (c + chiBase < 5 * Kp) row_store(c + chiBase, acc2);
  } else if (c >= chiBase && c < chiBase + Kp) {
    sp.chi2[c - chiBase] = acc;
    sp.n[c - chiBase] = accN;
  }
  __syncthreads();
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

__device__ void sort_candidates(EmShared &S, const SplitState &sp) {
  // getSplitCandidates (Splitter.h:1103-1117): descending chi-square, equal
  // values keep index order
  int n = int(sp.K);
  for (int i = 0; i < n; ++i) { S.candIdx[i] = i; S.candChi[i] = sp.chi2[i]; }
  for (int i = 1; i < n; ++i) {
    int ci = S.candIdx[i];
    float cv = S.candChi[i];
    int j = i - 1;
    while (j >= 0 && cv > S.candChi[j]) { S.candIdx[j + 1] = S.candIdx[j]; S.candChi[j + 1] = S.candChi[j]; --j; }
    S.candIdx[j + 1] = ci;
    S.candChi[j + 1] = cv;
  }
  S.numCands = n;
}

// PerformMerging (Merger.h:67-89, 218-279): all pair costs in parallel, then
// the first minimum in (i, j) scan order below the threshold, as the smallest
// (cost, i, j) over the block's threads.  A region's merging was bound by the
// costs' double-precision functions and their table searches and by one
// thread's scan of the pairs: 1.3 M cycles per region with 23 to 30 lobes, now
// 0.3 M (fourth frame of 2,097,152 samples, whose EM launch 4.3 -> 3.1 ms).
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
      for (int p = tid; p < pairs; p += kEmThreads) {
        // p -> (i, j), i < j
        int i = 0, rem = p;
        while (rem >= K - 1 - i) { rem -= K - 1 - i; ++i; }
        const int j = i + 1 + rem;
        S.cost[i][j] = merge_cost(S.vmm, i, j);
      }
    } else {
      // after merging lastJ into lastI (and moving the last component into
      // slot lastJ) only the pairs with those two slots have new operands; a
      // pair's cost depends on its two components alone, so the others keep
      // the bits a full recomputation would give
      const int moved = lastJ < K ? 1 : 0;  // lastJ was not the last slot
      for (int t = tid; t < (1 + moved) * K; t += kEmThreads) {
        const int a = t < K ? lastI : lastJ, b = t < K ? t : t - K;
        if (b == a || (a == lastJ && b == lastI)) continue;  // (lastI, lastJ) is in the first row
        const int i = a < b ? a : b, j = a < b ? b : a;
        S.cost[i][j] = merge_cost(S.vmm, i, j);
      }
    }
    __syncthreads();
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
    if (tid == 0) {
      for (int w = 1; w < kEmThreads / 32; ++w) best = warpBest[w] < best ? warpBest[w] : best;
      const bool found = best != ~0ull;
      const int ci = int(uint32_t(best)) / kMaxK, cj = int(uint32_t(best)) % kMaxK;
      if (found) {
        VMMState &v = S.vmm;
        V3 muI = mk(v.mx[ci], v.my[ci], v.mz[ci]), muJ = mk(v.mx[cj], v.my[cj], v.mz[cj]);
        float wI = v.w[ci], wJ = v.w[cj];
        vmm_merge(v, ci, cj);
        V3 muK = mk(v.mx[ci], v.my[ci], v.mz[ci]);
        split_merge_stats(S.split, ci, cj, wI, muI, wJ, muJ, v.w[ci], muK);
        suff_merge(S.suff, ci, cj);
        total++;
        lastI = ci;
        lastJ = cj;
      }
      mergeAgain = (found && S.vmm.K > cfg.laneWidth) ? 1 : 0;
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
    if (tid == 0) {
      sort_candidates(S, S.lsplit);
      for (int k = 0; k < kMaxK; ++k) S.mask[k] = 0;
      int numComp = int(S.vmm.K);
      for (int k = 0; k < numComp; ++k) {
        if (S.candChi[k] > cfg.splitThreshold && S.vmm.K < kMaxK) {
          bool ok = split_component(S.vmm, S.lsplit, S.temp, S.candIdx[k], cfg);
          S.mask[S.candIdx[k]] = 1;
          S.mask[S.vmm.K - 1] = 1;
          if (ok) S.splitCount++;
        }
      }
      if (S.splitCount > 0) suff_clear(S.temp, S.vmm.K);
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
      if (tid == 0) {
        for (int k = 0; k < kMaxK; ++k) S.mask[k] = 0;
        sort_candidates(S, S.split);
        int total = 0;
        for (int k = 0; k < S.numCands; ++k) {
          if (S.candChi[k] > cfg.splitThreshold && S.vmm.K < kMaxK) {
            split_component(S.vmm, S.split, S.suff, S.candIdx[k], cfg);
            S.mask[S.candIdx[k]] = 1;
            S.mask[S.vmm.K - 1] = 1;
            total++;
          }
        }
        S.report.splits += uint32_t(total);
        doRefit = (total > 0 && cfg.partialReFit && uint64_t(L.count) >= uint64_t(int64_t(cfg.minRefit))) ? 1 : 0;
        if (doRefit) {
          S.temp = S.suff;
          suff_clear(S.temp, S.vmm.K);
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
        if (threadIdx.x == 0) {
          S.vmm.pivot[0] = t.mean[0]; S.vmm.pivot[1] = t.mean[1]; S.vmm.pivot[2] = t.mean[2];
          valid = vmm_is_valid(S.vmm) ? 1u : 0u;
          afterSplit = 0;
          afterMerge = 0;
        }
      } else {
        if (threadIdx.x == 0 && cfg.parallax) {  // Field.h:476-482
          V3 shift = mk(S.vmm.pivot[0] - t.mean[0], S.vmm.pivot[1] - t.mean[1], S.vmm.pivot[2] - t.mean[2]);
          suff_parallax_shift(S.suff, S.vmm, shift);
          vmm_parallax_shift(S.vmm, shift);
        }
        __syncthreads();
        asm_update(S, L, cfg, afterSplit, afterMerge);
        if (threadIdx.x == 0)
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
