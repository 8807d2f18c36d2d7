// Guided queries: kd lookup, stochastic nearest-region choice, parallax shift
// of the region's mixture to the query point, cosine product, sampling and
// pdf evaluation (Field.h:109-145, KNN.h:22-28,134-148,
// VMMSurfaceSamplingDistribution.h:37-108, PAVMM.h:609-831).
//
// The arithmetic mirrors the reference's 8-wide SIMD lanes: per-lobe arithmetic
// is the reference's, and horizontal sums use shuffles in the vfloat8 reduce
// order (lobes j, j+8, j+16, j+24 summed in vector order, then the 8-lane tree).
// Per-object calls take a warp with lane k owning lobe k, batches several
// queries per warp with two or four lobes per lane.
#include <cuda_runtime.h>

#include "dqt.cuh"
#include "hg_table.h"
#include "launch.h"
#include "pgl_internal.h"

namespace pgl {




// (p[dim] >= pivot) goes right (KDTree.h:390-393); treelets give the same leaf.
__device__ __forceinline__ uint32_t kd_leaf(const FieldView &f, float p0, float p1, float p2) {
  uint32_t i = 0;
  KDNode n = f.nodes[0];
  while ((n.bits >> 30) != 3u) {
    uint32_t dim = n.bits >> 30;
    float c = dim == 0 ? p0 : (dim == 1 ? p1 : p2);
    i = (n.bits & 0x3FFFFFFFu) + (c >= n.split ? 1u : 0u);
    n = f.nodes[i];
  }
  return n.bits & 0x3FFFFFFFu;
}

// Returns the region to use, updating s1d (KNN.h:22-28, 134-148).
__device__ uint32_t choose_region(const FieldView &f, uint32_t leaf, float p0, float p1, float p2, float &s1d,
                                  int lane) {
  const Neighbours &nb = f.nbrs[leaf];
  uint32_t size = min(4u, nb.size);
  uint32_t sel = uint32_t(s1d * float(size));
  s1d = (s1d - float(sel) / float(size)) * float(size);
  sel = min(sel, size - 1);
  uint32_t key = 0xFFFFFFFFu;
  if (lane < 8) {
    V3 d = mk(nb.px[lane] - p0, nb.py[lane] - p1, nb.pz[lane] - p2);
    float dd = dot(d, d);
    key = (f2u(dd) & ~7u) | uint32_t(lane);
    if (nb.ids[lane] == ~0u) key = f2u(INFINITY);
  }
  // rank among the 8 keys (all finite keys are distinct)
  uint32_t rank = 0;
  for (int j = 0; j < 8; ++j) {
    uint32_t kj = __shfl_sync(0xFFFFFFFFu, key, j);
    float fj = u2f(kj), fk = u2f(key);
    rank += (fj < fk) ? 1u : 0u;
  }
  uint32_t hit = __ballot_sync(0xFFFFFFFFu, lane < 8 && rank == sel && key != f2u(INFINITY));
  int src = __ffs(hit) - 1;
  uint32_t chosenKey = __shfl_sync(0xFFFFFFFFu, key, src < 0 ? 0 : src);
  return nb.ids[chosenKey & 7u];
}

// The same choice by one thread (quadtree fields: a thread per query): the
// lowest neighbour slot whose key has rank `sel`, else slot 0's.
__device__ uint32_t choose_region_1(const FieldView &f, uint32_t leaf, float p0, float p1, float p2, float &s1d) {
  const Neighbours &nb = f.nbrs[leaf];
  uint32_t size = min(4u, nb.size);
  uint32_t sel = uint32_t(s1d * float(size));
  s1d = (s1d - float(sel) / float(size)) * float(size);
  sel = min(sel, size - 1);
  // 128-bit loads: 32 threads read 32 lines with each one
  uint32_t key[8], ids[8];
  const uint4 *pid = reinterpret_cast<const uint4 *>(nb.ids);
  const float4 *px = reinterpret_cast<const float4 *>(nb.px), *py = reinterpret_cast<const float4 *>(nb.py),
               *pz = reinterpret_cast<const float4 *>(nb.pz);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 id = pid[h];
    const float4 x = px[h], y = py[h], z = pz[h];
    const uint32_t idv[4] = {id.x, id.y, id.z, id.w};
    const float xv[4] = {x.x, x.y, x.z, x.w}, yv[4] = {y.x, y.y, y.z, y.w}, zv[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      V3 d = mk(xv[j] - p0, yv[j] - p1, zv[j] - p2);
      float dd = dot(d, d);
      ids[4 * h + j] = idv[j];
      key[4 * h + j] = (f2u(dd) & ~7u) | uint32_t(4 * h + j);
      if (idv[j] == ~0u) key[4 * h + j] = f2u(INFINITY);
    }
  }
  uint32_t chosen = ids[0];
  bool found = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t rank = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) rank += (u2f(key[k]) < u2f(key[j])) ? 1u : 0u;
    if (!found && rank == sel && key[j] != f2u(INFINITY)) {
      found = true;
      chosen = ids[j];  // a finite key's low bits are its slot
    }
  }
  return chosen;
}

// vfloat8 horizontal sum of lane values over the mixture: per group lane j
// sums lanes j, j+8, ... over cnt vectors, then the 8-lane tree.
__device__ __forceinline__ float lane_sum(float v, int cnt, int lane) {
  float acc = 0.0f;
  for (int q = 0; q < cnt; ++q) acc += __shfl_sync(0xFFFFFFFFu, v, (q * kLanes + (lane & 7)) & 31);
  acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 1);
  acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 2);
  acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 4);
  return __shfl_sync(0xFFFFFFFFu, acc, 0);
}

// Copy of the region's lobe with the parallax shift to the query point
// (parallax-aware mixtures only: VMMSurfaceSamplingDistribution.h:41-46).
__device__ __forceinline__ Lobe load_shifted(const VMMState &v, int lane, float p0, float p1, float p2,
                                             bool parallax) {
  Lobe L;
  L.w = v.w[lane]; L.kappa = v.kappa[lane]; L.norm = v.norm[lane]; L.e2k = v.e2k[lane];
  float dist = v.dist[lane];
  V3 mu = mk(v.mx[lane], v.my[lane], v.mz[lane]);
  V3 s = mk(v.pivot[0] - p0, v.pivot[1] - p1, v.pivot[2] - p2);
  V3 p = mu * dist + s;
  bool cond = (dist > 0.0f) && (dist >= -FLT_MAX) && (dist <= FLT_MAX);
  if (cond && parallax) mu = div3(p, length(p));
  L.mx = mu.x; L.my = mu.y; L.mz = mu.z;
  return L;
}

// the phase function fits (VMMPhaseFunctions.cpp), uploaded with the seed tables
static_assert(kHgLobes == kMaxProducts, "a distribution holds one product per lobe of the fit");
static __constant__ HgLobeFit c_hg[kHgFits][kHgLobes];

// PAVMM::product with a single lobe of weight `weight` (the cosine lobe, or a
// lobe of the phase function's fit), before the normalisation by the
// product's integral
__device__ __forceinline__ Lobe product_terms(const Lobe &L, V3 n, float kappa, float normalization, float weight) {
  V3 mu = mk(L.mx, L.my, L.mz);
  V3 nm = mu * L.kappa + n * kappa;
  float nk = sqrtf(dot(nm, nm));
  bool chk = nk > 1e-3f;
  nk = chk ? nk : 0.0f;
  nm = chk ? div3(nm, nk) : mu;
  float ne = fexp(-2.0f * nk);
  float nn = nk / (kTwoPiF * (1.0f - ne));
  nn = chk ? nn : kInv4Pi;
  float scale = (L.norm * normalization) / nn;
  float c0 = dot(mu, nm), c1 = dot(n, nm);
  float ev = fexp(L.kappa * (c0 - 1.0f) + kappa * (c1 - 1.0f));
  scale *= ev;
  scale *= L.w * weight;
  Lobe R;
  R.w = scale; R.kappa = nk; R.mx = nm.x; R.my = nm.y; R.mz = nm.z; R.norm = nn; R.e2k = ne;
  return R;
}
// the product; integral = the product's integral
__device__ __forceinline__ Lobe product_lobe(Lobe L, V3 n, float kappa, float normalization, float weight, int cnt,
                                             int lane, float &integral) {
  Lobe R = product_terms(L, n, kappa, normalization, weight);
  integral = lane_sum(lane < cnt * kLanes ? R.w : 0.0f, cnt, lane);
  R.w /= integral;
  return R;
}

// one lobe's term of the mixture's pdf in direction d
__device__ __forceinline__ float mixture_term(const Lobe &L, V3 d) {
  float ct = dot(d, mk(L.mx, L.my, L.mz));
  float cm1 = emin(ct - 1.0f, 0.0f);
  float ev = L.norm * fexp(L.kappa * cm1);
  return L.w * ev;
}
__device__ __forceinline__ float mixture_pdf(const Lobe &L, V3 d, int cnt, int lane) {
  const float t = mixture_term(L, d);
  return lane_sum(lane < cnt * kLanes ? t : 0.0f, cnt, lane);
}

__device__ V3 lobe_direction(float k, float e2k, V3 mu, float ux, float u1);
// PAVMM::sample (PAVMM.h:737-806)
__device__ V3 mixture_sample(const Lobe &L, int K, float ux, float uy, int lane) {
  // per-vector sums of the weights
  float g = L.w;
  g += __shfl_xor_sync(0xFFFFFFFFu, g, 1);
  g += __shfl_xor_sync(0xFFFFFFFFu, g, 2);
  g += __shfl_xor_sync(0xFFFFFFFFu, g, 4);
  float vecSum[4];
  for (int q = 0; q < 4; ++q) vecSum[q] = __shfl_sync(0xFFFFFFFFu, g, q * kLanes);
  uint32_t sv = 0, sc = 0;
  float searched = uy, sumW = 0.0f, cdf = 0.0f;
  uint32_t quot = uint32_t((K - 1) / kLanes), rem = uint32_t((K - 1) % kLanes);
  for (;;) {
    cdf = vecSum[sv];
    if (sumW + cdf >= searched || sv + 1 >= quot + 1) break;
    sumW += cdf;
    sv++;
  }
  uint32_t maxSel = (sv == quot) ? rem + 1 : kLanes;
  for (;;) {
    cdf = __shfl_sync(0xFFFFFFFFu, L.w, int(sv * kLanes + sc));
    if (sumW + cdf >= searched || sc + 1 >= maxSel) break;
    sumW += cdf;
    sc++;
  }
  float u1 = smin(1.0f - FLT_EPSILON, (searched - sumW) / cdf);
  int s = int(sv * kLanes + sc);
  float k = __shfl_sync(0xFFFFFFFFu, L.kappa, s), e2k = __shfl_sync(0xFFFFFFFFu, L.e2k, s);
  V3 mu = mk(__shfl_sync(0xFFFFFFFFu, L.mx, s), __shfl_sync(0xFFFFFFFFu, L.my, s), __shfl_sync(0xFFFFFFFFu, L.mz, s));
  return lobe_direction(k, e2k, mu, ux, u1);
}
// A direction of the chosen lobe (kappa k, e^{-2k}, mean mu) from the
// rescaled uniform u1 and ux (PAVMM.h:779-806)
__device__ V3 lobe_direction(float k, float e2k, V3 mu, float ux, float u1) {
  V3 d;
  if (k == 0.0f) {
    float z = 1.0f - 2.0f * u1;
    float r = sqrtf(smax(0.f, (1.0f - z * z)));
    float sp, cp;
    lib_sincosf(two_pi_times(ux), &sp, &cp);
    d = mk(r * cp, r * sp, z);
  } else {
    float ct = 1.f + (flog(1.0f + ((e2k - 1.f) * ux))) / k;
    ct = smin(1.0f, smax(ct, -1.f));
    float st = sqrtf(1.f - ct * ct);
    float phi = two_pi_times(u1);
    float sp, cp;
    lib_sincosf(phi, &sp, &cp);
    d = mk(st * cp, st * sp, ct);
  }
  return xfm(frame_of(mu, false), d);
}


// The Henyey-Greenstein product (VMMVolumeSamplingDistribution.h:54-80,
// VMMPhaseFunctions.h:45-57): the fit for |meanCosine|, li times each of its
// lobes (lobes of the fit's sign facing dir, else -dir); w = the products'
// integrals over their sum.
__device__ __forceinline__ void hg_products(const Lobe &li, V3 dir, float meanCosine, int cnt, int lane,
                                            Lobe h[kHgLobes], float w[kHgLobes]) {
  const float absG = fabsf(meanCosine);
  const float step = (kHgMaxMeanCosine - kHgMinMeanCosine) / float(kHgFits);
  int idx = int(floorf((absG - kHgMinMeanCosine) / step));
  idx = idx < kHgFits - 1 ? idx : kHgFits - 1;
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < kHgLobes; ++i) {
    const HgLobeFit fit = c_hg[idx][i];
    const V3 out = meanCosine * fit.meanCosine > 0.f ? dir : mk(-dir.x, -dir.y, -dir.z);
    h[i] = product_lobe(li, out, fit.kappa, fit.normalization, fit.weight, cnt, lane, w[i]);
    sum += w[i];
  }
#pragma unroll
  for (int i = 0; i < kHgLobes; ++i) w[i] /= sum;
}
// Sample of a weighted set of products: the first product whose running
// weight passes u.x, sampled with u.x rescaled into it
// (VMMVolumeSamplingDistribution.h:87-105); pdf = the weighted sum.
__device__ __forceinline__ V3 products_sample(const Lobe h[kHgLobes], const float w[kHgLobes], int np, int K, float ux,
                                              float uy, int lane, float &pdf) {
  float acc = 0.0f;
  int i = 0;
  for (; i < np - 1; ++i) {
    const float next = acc + w[i];
    if (next > ux) break;
    acc = next;
  }
  const Lobe g = i == 0 ? h[0] : (i == 1 ? h[1] : h[2]);
  const float wi = i == 0 ? w[0] : (i == 1 ? w[1] : w[2]);
  const V3 d = mixture_sample(g, K, (ux - acc) / wi, uy, lane);
  const int cnt = vec_count(K);
  pdf = 0.0f;
  for (int k = 0; k < np; ++k) pdf += w[k] * mixture_pdf(h[k], d, cnt, lane);
  return d;
}

// ---------------------------------------------------------------- quadtree regions
// SphereToSquareCylindrical::pointToDirection (SphereToSquare.h:40-55), with
// the host C library's cosf and sinf of the azimuth
__device__ V3 dqt_point_to_dir(float px, float py) {
  px = dqt_clamp(px, 0.f, 1.f);
  py = dqt_clamp(py, 0.f, 1.f);
  const float cosTheta = 2.0f * px - 1.0f;
  const float sinTheta = sqrtf(1.0f - cosTheta * cosTheta);
  float sinPhi, cosPhi;
  lib_sincosf_any(dqt_phi(py), &sinPhi, &cosPhi);
  return mk(dqt_clamp(sinTheta * cosPhi, -1.f, 1.f), dqt_clamp(sinTheta * sinPhi, -1.f, 1.f),
            dqt_clamp(cosTheta, -1.f, 1.f));
}
// samplePdf (DQT.h:62-72, :115-153): a stochastic descent that picks the
// left or right half by u.x and the lower or upper half by u.y, each
// rescaled into the chosen part; pdf = leaf weight / (root weight x leaf
// area) / 4 pi
__device__ float dqt_sample_pdf(const DqtNode *N, float ux, float uy, V3 &dir) {
  float span = 1.0f, x = 0.0f, y = 0.0f;
  // one division either way
  auto rescale = [](float t, float &u) {
    const bool first = u < t;
    u = (first ? u : u - t) / (first ? t : 1.0f - t);
    return first;
  };
  // a node's four children are one load each, and the chosen one's own child comes with it
  const auto node = [&](uint32_t i) {
    const uint2 v = *reinterpret_cast<const uint2 *>(&N[i]);
    return DqtNode{v.x, u2f(v.y)};
  };
  const DqtNode root = node(0);
  DqtNode at = root;
  while (at.child > 0) {
    span /= 2.0f;
    const DqtNode c0 = node(at.child), c1 = node(at.child + 1), c2 = node(at.child + 2), c3 = node(at.child + 3);
    const float wl = c0.weight + c2.weight, wr = c1.weight + c3.weight;
    const bool left = rescale(wl / (wl + wr), ux);
    if (!left) x += span;
    const DqtNode t = left ? c0 : c1, b = left ? c2 : c3;
    const bool top = rescale(t.weight / (t.weight + b.weight), uy);
    if (!top) y += span;
    at = top ? t : b;
  }
  float pdf = at.weight / (root.weight * span * span);
  const float px = x + ux * span, py = y + uy * span;
  pdf /= kDqtJacobian;
  dir = dqt_point_to_dir(px, py);
  return pdf;
}
// pdf (DQT.h:53-60, :155-159)
__device__ float dqt_pdf(const DqtNode *N, V3 d) {
  float px, py;
  dqt_dir_to_point(d.x, d.y, d.z, px, py);
  Box2 rect;
  const uint32_t i = dqt_query(N, px, py, rect);
  const float p = N[i].weight / (N[0].weight * rect.area()) / kDqtJacobian;
  return smin(FLT_MAX, p);
}
// A guided query on a quadtree region (DQTSurfaceSamplingDistribution.h /
// DQTVolumeSamplingDistribution.h: no products, pdfLi = pdf); lane 0 writes.
__device__ void dqt_query_out(const FieldView &f, uint32_t reg, uint32_t leaf, float ux, float uy, QueryOut &o) {
  if (!f.dqtHeads[reg].valid) return;
  const DqtNode *N = f.dqtNodes + size_t(reg) * f.dqtStride;
  V3 d;
  o.pdf = dqt_sample_pdf(N, ux, uy, d);
  o.ok = 1;
  o.id = leaf;
  o.dx = d.x;
  o.dy = d.y;
  o.dz = d.z;
  o.pdfLi = dqt_pdf(N, d);
}

// ---------------------------------------------------------------- several queries per warp
// A group of 8 * kH lanes per query.  With kH = 1 (four queries per warp) lane j
// holds lobes j, j + 8, j + 16 and j + 24, with kH = 2 (two per warp) lobes j
// and j + 16: lane j of every lobe vector (vfloat8) sits in a lane whose low
// three bits are j.  So the sums over the mixture keep the warp-per-query order
// (per vector lane over the vectors, then the 8-lane tree).
// Shuffles stay inside the group (its width, its lane mask): groups of one warp
// may take different paths.
template <int kH>
constexpr int kSlots = 4 / kH;  // lobes per lane
template <int kH>
struct Group {
  int j;        // lane of the group
  unsigned gm;  // its lane mask
  __device__ __forceinline__ explicit Group(int lane)
      : j(lane & (8 * kH - 1)), gm((kH == 1 ? 0xFFu : 0xFFFFu) << (lane & (32 - 8 * kH))) {}
  template <typename T>
  __device__ __forceinline__ T from(T v, int src) const {
    return __shfl_sync(gm, v, src, 8 * kH);
  }
  // the 8-lane tree: all eight lanes end with the same bits (each step adds the
  // same two numbers on both sides)
  __device__ __forceinline__ float tree(float v) const {
    v += __shfl_xor_sync(gm, v, 1, 8);
    v += __shfl_xor_sync(gm, v, 2, 8);
    v += __shfl_xor_sync(gm, v, 4, 8);
    return v;
  }
  // the sum over the mixture; lobes past its last vector count +0, which changes
  // no bit of a sum that started at +0
  __device__ __forceinline__ float sum(const float v[kSlots<kH>]) const {
    float acc = 0.0f;
    if constexpr (kH == 1) {
#pragma unroll
      for (int q = 0; q < kSlots<kH>; ++q) acc += v[q];
    } else {
      // vectors 0 and 1 sit in the two halves and add in either order, vectors 2 and 3 in theirs
      acc = (acc + v[0]) + __shfl_xor_sync(gm, v[0], 8, 16);
      const float o = __shfl_xor_sync(gm, v[1], 8, 16);
      acc = j < 8 ? (acc + v[1]) + o : (acc + o) + v[1];
    }
    return tree(acc);
  }
};
template <int kH>
struct LobeSet {
  Lobe l[kSlots<kH>];
};
// is slot q of this lane in one of the mixture's cnt lobe vectors?
template <int kH>
__device__ __forceinline__ bool holds(const Group<kH> &G, int q, int cnt) {
  return q * kH + (kH == 1 ? 0 : G.j >> 3) < cnt;
}
// the lobe vectors of the mixture (the other slots hold zeros)
template <int kH>
__device__ __forceinline__ LobeSet<kH> load_shifted_g(const Group<kH> &G, const VMMState &v, float p0, float p1, float p2,
                                                      bool parallax, int cnt) {
  LobeSet<kH> L;
#pragma unroll
  for (int q = 0; q < kSlots<kH>; ++q) {
    L.l[q] = Lobe{};
    if (holds(G, q, cnt)) L.l[q] = load_shifted(v, q * 8 * kH + G.j, p0, p1, p2, parallax);
  }
  return L;
}
template <int kH>
__device__ __forceinline__ LobeSet<kH> product_lobe_g(const Group<kH> &G, const LobeSet<kH> &L, V3 n, float kappa,
                                                      float normalization, float weight, int cnt, float &integral) {
  LobeSet<kH> R;
  float w[kSlots<kH>];
#pragma unroll
  for (int q = 0; q < kSlots<kH>; ++q) {
    R.l[q] = Lobe{};
    if (holds(G, q, cnt)) R.l[q] = product_terms(L.l[q], n, kappa, normalization, weight);
    w[q] = R.l[q].w;
  }
  integral = G.sum(w);
#pragma unroll
  for (int q = 0; q < kSlots<kH>; ++q)
    if (holds(G, q, cnt)) R.l[q].w /= integral;
  return R;
}
template <int kH>
__device__ __forceinline__ float mixture_pdf_g(const Group<kH> &G, const LobeSet<kH> &L, V3 d, int cnt) {
  float t[kSlots<kH>];
#pragma unroll
  for (int q = 0; q < kSlots<kH>; ++q) t[q] = holds(G, q, cnt) ? mixture_term(L.l[q], d) : 0.0f;
  return G.sum(t);
}
// PAVMM::sample (PAVMM.h:737-806) by a group: the lobe that uy picks and uy
// rescaled into it; the direction in the lobe is lobe_direction's.  Both
// searches run without branches, so the groups of a warp stay together.
struct PickedLobe {
  float kappa, e2k, u1;
  V3 mu;
};
template <int kH>
__device__ __forceinline__ PickedLobe mixture_pick_g(const Group<kH> &G, const LobeSet<kH> &L, int K, float uy) {
  const int cnt = vec_count(K);
  const uint32_t quot = uint32_t((K - 1) / kLanes), rem = uint32_t((K - 1) % kLanes);
  // per-vector sums of the weights (vectors past the mixture's last are never searched)
  uint32_t sv = 0, sc = 0;
  float sumW = 0.0f, cdf = 0.0f;
  bool done = false;
#pragma unroll
  for (int q = 0; q < kSlots<kH>; ++q) {
    if (q * kH >= cnt) continue;
    const float t = G.tree(L.l[q].w);
#pragma unroll
    for (int h = 0; h < kH; ++h) {
      const float g = kH == 1 ? t : G.from(t, 8 * h);
      const uint32_t vec = uint32_t(q * kH + h);
      const bool stop = sumW + g >= uy || vec >= quot;
      sv = done ? sv : vec;
      sumW = done || stop ? sumW : sumW + g;
      done = done || stop;
    }
  }
  // the picked vector: the slot that its lanes hold it in, and the first of those lanes
  const uint32_t slot = sv / kH;
  const int first = kH == 1 ? 0 : int(sv % kH) * 8;
  const auto held = [&](auto field) {
    float r = L.l[0].*field;
#pragma unroll
    for (int q = 1; q < kSlots<kH>; ++q) r = slot == uint32_t(q) ? L.l[q].*field : r;
    return r;
  };
  const float vw = held(&Lobe::w);
  const uint32_t maxSel = (sv == quot) ? rem + 1 : kLanes;
  done = false;
#pragma unroll
  for (int c = 0; c < kLanes; ++c) {
    const float w = G.from(vw, first + c);
    const bool stop = sumW + w >= uy || uint32_t(c) + 1 >= maxSel;
    sc = done ? sc : uint32_t(c);
    cdf = done ? cdf : w;
    sumW = done || stop ? sumW : sumW + w;
    done = done || stop;
  }
  const int src = first + int(sc);
  PickedLobe r;
  r.u1 = smin(1.0f - FLT_EPSILON, (uy - sumW) / cdf);
  r.kappa = G.from(held(&Lobe::kappa), src);
  r.e2k = G.from(held(&Lobe::e2k), src);
  r.mu = mk(G.from(held(&Lobe::mx), src), G.from(held(&Lobe::my), src), G.from(held(&Lobe::mz), src));
  return r;
}
// The directions of a block's kN picked lobes, a thread per lobe (groups would
// run lobe_direction on one lobe with all their lanes: its logarithm, sine and
// cosine, and frame cost a sixth of a surface query).  Every thread of the block
// calls it; `writer` threads hand in the lobe of slot `i`, every thread gets the
// direction of slot `i`.  1,048,576 surface queries 706 -> 635 us, 262,147 with
// the phase function 411 -> 377 us, 1,000,003 vertices 911 -> 877 us.
template <int kN>
struct DirectionSlots {
  float kappa[kN], e2k[kN], u1[kN], ux[kN], x[kN], y[kN], z[kN];
};
template <int kN>
__device__ __forceinline__ V3 block_direction(DirectionSlots<kN> &S, int i, bool writer, const PickedLobe &p, float ux) {
  if (writer) {
    S.kappa[i] = p.kappa;
    S.e2k[i] = p.e2k;
    S.u1[i] = p.u1;
    S.ux[i] = ux;
    S.x[i] = p.mu.x;
    S.y[i] = p.mu.y;
    S.z[i] = p.mu.z;
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < kN) {
    const V3 d = lobe_direction(S.kappa[t], S.e2k[t], mk(S.x[t], S.y[t], S.z[t]), S.ux[t], S.u1[t]);
    S.x[t] = d.x;
    S.y[t] = d.y;
    S.z[t] = d.z;
  }
  __syncthreads();
  return mk(S.x[i], S.y[i], S.z[i]);
}
// choose_region by a group: lane j ranks neighbour j
__device__ uint32_t choose_region_g(const FieldView &f, uint32_t leaf, float p0, float p1, float p2, float &s1d,
                                    int j, int lane, unsigned gm) {
  const Neighbours &nb = f.nbrs[leaf];
  uint32_t size = min(4u, nb.size);
  uint32_t sel = uint32_t(s1d * float(size));
  s1d = (s1d - float(sel) / float(size)) * float(size);
  sel = min(sel, size - 1);
  V3 d = mk(nb.px[j] - p0, nb.py[j] - p1, nb.pz[j] - p2);
  float dd = dot(d, d);
  uint32_t key = (f2u(dd) & ~7u) | uint32_t(j);
  if (nb.ids[j] == ~0u) key = f2u(INFINITY);
  uint32_t rank = 0;
  for (int jj = 0; jj < 8; ++jj) {
    uint32_t kj = __shfl_sync(gm, key, jj, 8);
    rank += (u2f(kj) < u2f(key)) ? 1u : 0u;
  }
  const uint32_t hit = (__ballot_sync(gm, rank == sel && key != f2u(INFINITY)) >> (lane & 24)) & 0xFFu;
  int src = __ffs(hit) - 1;
  uint32_t chosenKey = __shfl_sync(gm, key, src < 0 ? 0 : src, 8);
  return nb.ids[chosenKey & 7u];
}

// Init of a group's query: false when it is outside the field or its region is
// not valid; else its kd leaf, region and rescaled s1d.
struct GroupInit {
  uint32_t leaf, reg;
  float s1d;
  bool ok;
};
template <typename Q>
__device__ __forceinline__ GroupInit init_g(const FieldView &f, const Q &q, int lane) {
  GroupInit r{0, 0, q.s1d, false};
  const bool inside = f.iteration > 0 && q.px >= f.bounds[0] && q.px <= f.bounds[3] && q.py >= f.bounds[1] &&
                      q.py <= f.bounds[4] && q.pz >= f.bounds[2] && q.pz <= f.bounds[5];
  if (inside) {
    r.leaf = r.reg = kd_leaf(f, q.px, q.py, q.pz);
    if (f.knn && r.s1d >= 0.f) r.reg = choose_region_g(f, r.leaf, q.px, q.py, q.pz, r.s1d, lane & 7, lane, 0xFFu << (lane & 24));
    r.ok = f.regions[r.reg].valid != 0;
  }
  return r;
}

// Blocks of a batch that fills the chip, and of one that does not: a small batch
// takes one query's latency, which is shorter with few warps on an SM, with the
// registers of few blocks and without the exchange of directions; one with the
// phase function with a warp per query.  Surface and volume queries and vertices
// take the small form while its blocks run in one wave (84 registers: ten blocks of
// eight queries per SM, 12,160 queries; 72: fourteen, 17,024 vertices): it stays
// ahead up to there and loses its gain with a second wave.  With the phase
// function (one wave is 4,864) the forms cross before that.  Launch by launch, us,
// large form / small:
//   surface     777 10.8 / 9.9   8,192 12.0 / 11.2  12,000 13.8 / 12.5  13,000 13.9 / 18.6  16,384 16.0 / 19.4
//   vertices    777 15.0 / 14.3  8,000 16.1 / 15.6  12,000 18.6 / 17.3  16,384 21.8 / 20.8  18,000 22.4 / 28.2
//   phase fn.   300 11.7 / 8.3   3,000 12.5 / 10.0   4,096 12.9 / 12.3   4,400 12.9 / 13.2   5,200 14.6 / 16.2
// (1,048,576 surface queries 635 / 706 us without the exchange, in blocks of 256).
constexpr int kQueryThreads = 256, kQueryBlocks = 4, kFewThreads = 64, kFewBlocks = 4;
constexpr uint32_t kFewQueries = 12160, kFewVertices = 16384, kFewHg = 4096;
// Batched volume guided queries with the Henyey-Greenstein product, two per
// warp: Init + product with the phase function's fit + SamplePDF (+ pdfLi).
// The mixture and its three products are live together, so a lane holds two
// lobes of each; 64 registers for four blocks per SM.  262,147 queries: 507 us
// with a warp per query, 377 us so (383 at 80 registers, 387 in blocks of 128
// threads, 490 in blocks of 512).
__global__ void __launch_bounds__(kQueryThreads, kQueryBlocks)
query_hg_kernel(QueryParams P, const QueryIn *in, QueryOut *out, uint32_t n) {
  __shared__ DirectionSlots<kQueryThreads / 16> slots;
  const uint32_t gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const int lane = threadIdx.x & 31;
  const Group<2> G(lane);
  const FieldView &f = P.f;
  const QueryIn q = in[min(gid, n - 1)];
  const GroupInit init = init_g(f, q, lane);
  LobeSet<2> li, h[kHgLobes];
  float w[kHgLobes], ux = 0.0f;
  PickedLobe p{};
  int cnt = 0;
  if (init.ok) {  // an untrained field has no regions to read
    const VMMState &v = f.regions[init.reg].vmm;
    const int K = int(v.K);
    cnt = vec_count(K);
    li = load_shifted_g<2>(G, v, q.px, q.py, q.pz, f.parallax != 0, cnt);
    const float meanCosine = P.hgMeanCosine[gid < n ? gid : n - 1];
    const float step = (kHgMaxMeanCosine - kHgMinMeanCosine) / float(kHgFits);
    int idx = int(floorf((fabsf(meanCosine) - kHgMinMeanCosine) / step));
    idx = idx < kHgFits - 1 ? idx : kHgFits - 1;
    const V3 dir = mk(q.nx, q.ny, q.nz);
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kHgLobes; ++i) {  // hg_products
      const HgLobeFit fit = c_hg[idx][i];
      const V3 to = meanCosine * fit.meanCosine > 0.f ? dir : mk(-dir.x, -dir.y, -dir.z);
      h[i] = product_lobe_g<2>(G, li, to, fit.kappa, fit.normalization, fit.weight, cnt, w[i]);
      sum += w[i];
    }
#pragma unroll
    for (int i = 0; i < kHgLobes; ++i) w[i] /= sum;
    // products_sample
    float acc = 0.0f;
    int i = 0;
    for (; i < kHgLobes - 1; ++i) {
      const float next = acc + w[i];
      if (next > q.ux) break;
      acc = next;
    }
    const LobeSet<2> g = i == 0 ? h[0] : (i == 1 ? h[1] : h[2]);
    const float wi = i == 0 ? w[0] : (i == 1 ? w[1] : w[2]);
    p = mixture_pick_g<2>(G, g, K, q.uy);
    ux = (q.ux - acc) / wi;
  }
  const V3 d = block_direction(slots, threadIdx.x >> 4, G.j == 0, p, ux);
  QueryOut o;
  o.ok = init.ok ? 1u : 0u;
  o.id = init.ok ? init.leaf : 0u;
  o.s1d = init.s1d;
  o.dx = o.dy = o.dz = 0.0f;
  o.pdf = o.pdfLi = 0.0f;
  if (init.ok) {
#pragma unroll
    for (int k = 0; k < kHgLobes; ++k) o.pdf += w[k] * mixture_pdf_g<2>(G, h[k], d, cnt);
    o.dx = d.x;
    o.dy = d.y;
    o.dz = d.z;
    o.pdfLi = mixture_pdf_g<2>(G, li, d, cnt);
  }
  if (gid < n && G.j == 0) out[gid] = o;
}

// The same for a batch that does not fill the chip: a warp per query, a lobe per
// lane, so that a query's chain is one lobe's work.
__global__ void query_hg_few_kernel(QueryParams P, const QueryIn *in, QueryOut *out, uint32_t n) {
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= n) return;
  const QueryIn q = in[gw];
  const FieldView &f = P.f;
  QueryOut o;
  o.ok = 0; o.id = 0; o.s1d = q.s1d; o.dx = o.dy = o.dz = 0.0f; o.pdf = 0.0f; o.pdfLi = 0.0f;
  bool inside = f.iteration > 0 && q.px >= f.bounds[0] && q.px <= f.bounds[3] && q.py >= f.bounds[1] &&
                q.py <= f.bounds[4] && q.pz >= f.bounds[2] && q.pz <= f.bounds[5];
  if (inside) {
    uint32_t leaf = kd_leaf(f, q.px, q.py, q.pz);
    uint32_t reg = leaf;
    float s1d = q.s1d;
    if (f.knn && s1d >= 0.f) reg = choose_region(f, leaf, q.px, q.py, q.pz, s1d, lane);
    o.s1d = s1d;
    const RegionDir &R = f.regions[reg];
    if (R.valid) {
      const int K = int(R.vmm.K), cnt = vec_count(K);
      Lobe li = load_shifted(R.vmm, lane, q.px, q.py, q.pz, f.parallax != 0);
      Lobe h[kHgLobes];
      float w[kHgLobes];
      hg_products(li, mk(q.nx, q.ny, q.nz), P.hgMeanCosine[gw], cnt, lane, h, w);
      const V3 d = products_sample(h, w, kHgLobes, K, q.ux, q.uy, lane, o.pdf);
      o.ok = 1;
      o.id = leaf;
      o.dx = d.x; o.dy = d.y; o.dz = d.z;
      o.pdfLi = mixture_pdf(li, d, cnt, lane);
    }
  }
  if (lane == 0) out[gw] = o;
}

// Batched guided queries, four per warp: Init + optional cosine product
// (surface) + SamplePDF (+ pdfLi).  Issue bound at about three quarters of the
// issue rate; 64 registers for four blocks per SM.  1,048,576 queries: 818 us
// with searches by branches, FP64 in lobe_direction, divisions one by one and
// the rsqrt table in constant memory (its lookups went one by one), 635 us so
// (687 at 80 registers, 660 at 48, 669 in blocks of 128 threads).
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
query_g_kernel(QueryParams P, const QueryIn *in, QueryOut *out, uint32_t n) {
  const uint32_t gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int lane = threadIdx.x & 31;
  const Group<1> G(lane);
  const QueryIn q = in[min(gid, n - 1)];
  const FieldView &f = P.f;
  const GroupInit init = init_g(f, q, lane);
  LobeSet<1> li, g;
  PickedLobe p{};
  int cnt = 0;
  if (init.ok) {  // an untrained field has no regions to read
    const VMMState &v = f.regions[init.reg].vmm;
    const int K = int(v.K);
    cnt = vec_count(K);
    li = load_shifted_g<1>(G, v, q.px, q.py, q.pz, f.parallax != 0, cnt);
    float integral;
    g = li;
    if (P.cosine) g = product_lobe_g<1>(G, li, mk(q.nx, q.ny, q.nz), P.cosKappa, P.cosNorm, 1.0f, cnt, integral);
    p = mixture_pick_g<1>(G, g, K, q.uy);
  }
  const float ux = (q.ux - 0.0f) / 1.0f;
  V3 d;
  if constexpr (kThreads == kFewThreads) {
    d = lobe_direction(p.kappa, p.e2k, p.mu, ux, p.u1);
  } else {
    __shared__ DirectionSlots<kThreads / 8> slots;
    d = block_direction(slots, threadIdx.x >> 3, G.j == 0, p, ux);
  }
  QueryOut o;
  o.ok = 0; o.id = 0; o.s1d = init.s1d; o.dx = o.dy = o.dz = 0.0f; o.pdf = 0.0f; o.pdfLi = 0.0f;
  if (init.ok) {
    o.ok = 1;
    o.id = init.leaf;
    o.dx = d.x; o.dy = d.y; o.dz = d.z;
    o.pdf = 0.0f + 1.0f * mixture_pdf_g<1>(G, g, d, cnt);
    o.pdfLi = mixture_pdf_g<1>(G, li, d, cnt);
  }
  if (gid < n && G.j == 0) out[gid] = o;
}
// Batched path-vertex query, four per warp: Init + cosine product once, then
// one SamplePDF per 2D random number on the same distribution (the sampled
// distribution is not changed by sampling: VMMSurfaceSamplingDistribution.h:67-103),
// as a renderer does per vertex and openpgl_bench's lookup loop does per
// initialised distribution (openpgl_bench.cpp:343-362).  The group picks the
// four lobes one after the other, and the block finds all their directions at
// once.  1,000,003 vertices: 1,838 us with four runs through lobe_direction per
// vertex, 877 us so.
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
query_s4_g_kernel(QueryParams P, const QueryInS4 *in, QueryOutS4 *out, uint32_t n) {
  static_assert(kVertexSamples == 4, "two lanes of a group per sample");
  const uint32_t gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int lane = threadIdx.x & 31;
  const Group<1> G(lane);
  const QueryInS4 &q = in[min(gid, n - 1)];
  const FieldView &f = P.f;
  struct {
    float px, py, pz, s1d;
  } at = {q.px, q.py, q.pz, q.s1d};
  const GroupInit init = init_g(f, at, lane);
  const int mine = G.j & 3;
  const float ux = q.u[mine][0], uyMine = q.u[mine][1];
  LobeSet<1> g;
  PickedLobe p{};
  int cnt = 0;
  if (init.ok) {  // an untrained field has no regions to read
    const VMMState &v = f.regions[init.reg].vmm;
    const int K = int(v.K);
    cnt = vec_count(K);
    g = load_shifted_g<1>(G, v, q.px, q.py, q.pz, f.parallax != 0, cnt);
    float integral;
    if (P.cosine) g = product_lobe_g<1>(G, g, mk(q.nx, q.ny, q.nz), P.cosKappa, P.cosNorm, 1.0f, cnt, integral);
#pragma unroll 1
    for (int k = 0; k < kVertexSamples; ++k) {
      const PickedLobe t = mixture_pick_g<1>(G, g, K, G.from(uyMine, k));
      if (k == mine) p = t;
    }
  }
  V3 d;
  if constexpr (kThreads == kFewThreads) {
    d = lobe_direction(p.kappa, p.e2k, p.mu, (ux - 0.0f) / 1.0f, p.u1);
  } else {
    __shared__ DirectionSlots<kThreads / 2> slots;
    d = block_direction(slots, (threadIdx.x >> 3) * 4 + mine, G.j < kVertexSamples, p, (ux - 0.0f) / 1.0f);
  }
  float pdf = 0.0f;  // of sample `mine`
  if (init.ok) {
#pragma unroll 1
    for (int k = 0; k < kVertexSamples; ++k) {
      const V3 dk = mk(G.from(d.x, k), G.from(d.y, k), G.from(d.z, k));
      const float t = 0.0f + 1.0f * mixture_pdf_g<1>(G, g, dk, cnt);
      if (k == mine) pdf = t;
    }
  } else {
    d = mk(0.0f, 0.0f, 0.0f);
  }
  if (gid >= n) return;
  QueryOutS4 &o = out[gid];
  if (G.j == 0) {
    o.ok = init.ok ? 1u : 0u;
    o.id = init.ok ? init.leaf : 0u;
    o.s1d = init.s1d;
  }
  if (G.j < kVertexSamples) {
    o.s[mine][0] = d.x;
    o.s[mine][1] = d.y;
    o.s[mine][2] = d.z;
    o.s[mine][3] = pdf;
  }
}


// Batched guided queries on a quadtree field: a thread per query (a
// quadtree's descent has no lobes to spread over a warp).  Latency bound, so as
// many threads as fit.  1,048,576 queries: 206 us with the angle, its sine and the
// direction's turn in double, the neighbours in 33 loads and two loads one after
// the other per level, 160 us without those, 135 us at 32 registers; vertices of
// four samples 643, 461 and (at 40) 404 us.
__global__ void __launch_bounds__(256, 8) query_dqt_kernel(QueryParams P, const QueryIn *in, QueryOut *out, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const QueryIn q = in[i];
  const FieldView &f = P.f;
  QueryOut o;
  o.ok = 0; o.id = 0; o.s1d = q.s1d; o.dx = o.dy = o.dz = 0.0f; o.pdf = 0.0f; o.pdfLi = 0.0f;
  const bool inside = f.iteration > 0 && q.px >= f.bounds[0] && q.px <= f.bounds[3] && q.py >= f.bounds[1] &&
                      q.py <= f.bounds[4] && q.pz >= f.bounds[2] && q.pz <= f.bounds[5];
  if (inside) {
    const uint32_t leaf = kd_leaf(f, q.px, q.py, q.pz);
    uint32_t reg = leaf;
    float s1d = q.s1d;
    if (f.knn && s1d >= 0.f) reg = choose_region_1(f, leaf, q.px, q.py, q.pz, s1d);
    o.s1d = s1d;
    dqt_query_out(f, reg, leaf, q.ux, q.uy, o);
  }
  out[i] = o;
}
__global__ void query_s4_dqt_kernel(QueryParams P, const QueryInS4 *in, QueryOutS4 *out, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const QueryInS4 q = in[i];
  const FieldView &f = P.f;
  QueryOutS4 o;
  o.ok = 0;
  o.id = 0;
  o.s1d = q.s1d;
#pragma unroll
  for (int k = 0; k < kVertexSamples; ++k) o.s[k][0] = o.s[k][1] = o.s[k][2] = o.s[k][3] = 0.0f;
  const bool inside = f.iteration > 0 && q.px >= f.bounds[0] && q.px <= f.bounds[3] && q.py >= f.bounds[1] &&
                      q.py <= f.bounds[4] && q.pz >= f.bounds[2] && q.pz <= f.bounds[5];
  if (inside) {
    const uint32_t leaf = kd_leaf(f, q.px, q.py, q.pz);
    uint32_t reg = leaf;
    float s1d = q.s1d;
    if (f.knn && s1d >= 0.f) reg = choose_region_1(f, leaf, q.px, q.py, q.pz, s1d);
    o.s1d = s1d;
    if (f.dqtHeads[reg].valid) {
      const DqtNode *N = f.dqtNodes + size_t(reg) * f.dqtStride;
      for (int k = 0; k < kVertexSamples; ++k) {
        V3 d;
        o.s[k][3] = dqt_sample_pdf(N, q.u[k][0], q.u[k][1], d);
        o.s[k][0] = d.x;
        o.s[k][1] = d.y;
        o.s[k][2] = d.z;
      }
      o.ok = 1;
      o.id = leaf;
    }
  }
  out[i] = o;
}

// ---------------------------------------------------------------- per-object path
// State of one SurfaceSamplingDistribution / VolumeSamplingDistribution on the
// device: the shifted mixture (for IncomingRadiancePDF) and the product one.

__global__ void ssd_init_kernel(FieldView f, float px, float py, float pz, float s1dIn, SSDState *st, SSDResult *res) {
  const int lane = threadIdx.x & 31;
  SSDResult r{0, 0, s1dIn, 0, 0, 0, 0};
  bool inside = f.iteration > 0 && px >= f.bounds[0] && px <= f.bounds[3] && py >= f.bounds[1] && py <= f.bounds[4] &&
                pz >= f.bounds[2] && pz <= f.bounds[5];
  if (inside) {
    uint32_t leaf = kd_leaf(f, px, py, pz);
    uint32_t reg = leaf;
    float s1d = s1dIn;
    if (f.knn && s1d >= 0.f) reg = choose_region(f, leaf, px, py, pz, s1d, lane);
    r.s1d = s1d;
    const RegionDir &R = f.regions[reg];
    if (f.dqt) {  // the quadtree is read from the field when sampled
      if (f.dqtHeads[reg].valid) {
        if (lane == 0) st->region = reg;
        r.ok = 1;
        r.id = leaf;
      }
    } else if (R.valid) {
      Lobe li = load_shifted(R.vmm, lane, px, py, pz, f.parallax != 0);
      st->li[lane] = li;
      st->g[lane] = li;
      if (lane == 0) {
        st->K = R.vmm.K;
        st->numProducts = 0;
      }
      r.ok = 1;
      r.id = leaf;
    }
  }
  if (lane == 0) *res = r;
}
__global__ void ssd_cosine_kernel(SSDState *st, float nx, float ny, float nz, float cosKappa, float cosNorm) {
  const int lane = threadIdx.x & 31;
  const int cnt = vec_count(int(st->K));
  float integral;
  Lobe g = product_lobe(st->g[lane], mk(nx, ny, nz), cosKappa, cosNorm, 1.0f, cnt, lane, integral);
  __syncwarp();
  st->g[lane] = g;
}
__global__ void ssd_hg_kernel(SSDState *st, float dx, float dy, float dz, float meanCosine) {
  const int lane = threadIdx.x & 31;
  const int cnt = vec_count(int(st->K));
  Lobe h[kHgLobes];
  float w[kHgLobes];
  hg_products(st->li[lane], mk(dx, dy, dz), meanCosine, cnt, lane, h, w);
#pragma unroll
  for (int i = 0; i < kHgLobes; ++i) st->h[i][lane] = h[i];
  if (lane == 0) {
    for (int i = 0; i < kHgLobes; ++i) st->hw[i] = w[i];
    st->numProducts = kHgLobes;
  }
}
__global__ void ssd_sample_kernel(const SSDState *st, float ux, float uy, int withPdf, SSDResult *res) {
  const int lane = threadIdx.x & 31;
  const int K = int(st->K), cnt = vec_count(K);
  V3 d;
  float pdf = 0.0f;
  if (st->numProducts > 0) {
    Lobe h[kHgLobes];
    float w[kHgLobes];
#pragma unroll
    for (int i = 0; i < kHgLobes; ++i) {
      h[i] = st->h[i][lane];
      w[i] = st->hw[i];
    }
    d = products_sample(h, w, int(st->numProducts), K, ux, uy, lane, pdf);
  } else {
    Lobe g = st->g[lane];
    d = mixture_sample(g, K, (ux - 0.0f) / 1.0f, uy, lane);
    pdf = withPdf ? 0.0f + 1.0f * mixture_pdf(g, d, cnt, lane) : 0.0f;
  }
  if (lane == 0) {
    res->dx = d.x; res->dy = d.y; res->dz = d.z; res->pdf = pdf;
  }
}
__global__ void ssd_pdf_kernel(const SSDState *st, float dx, float dy, float dz, int li, SSDResult *res) {
  const int lane = threadIdx.x & 31;
  const int cnt = vec_count(int(st->K));
  const V3 d = mk(dx, dy, dz);
  float pdf;
  if (li) {
    pdf = mixture_pdf(st->li[lane], d, cnt, lane);
  } else if (st->numProducts > 0) {
    pdf = 0.0f;
    for (uint32_t k = 0; k < st->numProducts; ++k) pdf += st->hw[k] * mixture_pdf(st->h[k][lane], d, cnt, lane);
  } else {
    pdf = 0.0f + 1.0f * mixture_pdf(st->g[lane], d, cnt, lane);
  }
  if (lane == 0) res->pdf = pdf;
}

// Per-object Sample / SamplePDF / PDF / IncomingRadiancePDF of a quadtree
// region (DQTSurfaceSamplingDistribution.h:28-45: pdfLi is the pdf).
__global__ void ssd_dqt_sample_kernel(FieldView f, const SSDState *st, float ux, float uy, SSDResult *res) {
  const DqtNode *N = f.dqtNodes + size_t(st->region) * f.dqtStride;
  V3 d;
  const float pdf = dqt_sample_pdf(N, ux, uy, d);
  res->dx = d.x;
  res->dy = d.y;
  res->dz = d.z;
  res->pdf = pdf;
}
__global__ void ssd_dqt_pdf_kernel(FieldView f, const SSDState *st, float dx, float dy, float dz, SSDResult *res) {
  const DqtNode *N = f.dqtNodes + size_t(st->region) * f.dqtStride;
  res->pdf = dqt_pdf(N, mk(dx, dy, dz));
}

// ---------------------------------------------------------------- launchers
PGL_DEFINE_TABLE_UPLOAD(query_upload_seed_tables)
cudaError_t query_upload_tables(const LibmTables &libm) {
  cudaError_t e = query_upload_seed_tables(libm);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_hg, kHgTable, sizeof(kHgTable));
}

cudaError_t launch_query(const QueryParams &p, const QueryIn *in, QueryOut *out, uint32_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned threads = 256;
  const auto blocks = [&](unsigned lanes, unsigned per) { return unsigned((uint64_t(n) * lanes + per - 1) / per); };
  count_launch();
  if (p.f.dqt) {
    query_dqt_kernel<<<unsigned((uint64_t(n) + threads - 1) / threads), threads, 0, s>>>(p, in, out, n);
    return cudaGetLastError();
  }
  if (p.hgMeanCosine) {
    if (n <= kFewHg)
      query_hg_few_kernel<<<blocks(32, kFewThreads), kFewThreads, 0, s>>>(p, in, out, n);
    else
      query_hg_kernel<<<blocks(16, kQueryThreads), kQueryThreads, 0, s>>>(p, in, out, n);
    return cudaGetLastError();
  }
  if (n <= kFewQueries)
    query_g_kernel<kFewThreads, kFewBlocks><<<blocks(8, kFewThreads), kFewThreads, 0, s>>>(p, in, out, n);
  else
    query_g_kernel<kQueryThreads, kQueryBlocks><<<blocks(8, kQueryThreads), kQueryThreads, 0, s>>>(p, in, out, n);
  return cudaGetLastError();
}
cudaError_t launch_query_s4(const QueryParams &p, const QueryInS4 *in, QueryOutS4 *out, uint32_t n,
                            cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned threads = 256;
  const auto blocks = [&](unsigned lanes, unsigned per) { return unsigned((uint64_t(n) * lanes + per - 1) / per); };
  count_launch();
  if (p.f.dqt) {
    query_s4_dqt_kernel<<<unsigned((uint64_t(n) + threads - 1) / threads), threads, 0, s>>>(p, in, out, n);
    return cudaGetLastError();
  }
  if (n <= kFewVertices)
    query_s4_g_kernel<kFewThreads, kFewBlocks><<<blocks(8, kFewThreads), kFewThreads, 0, s>>>(p, in, out, n);
  else
    query_s4_g_kernel<kQueryThreads, kQueryBlocks><<<blocks(8, kQueryThreads), kQueryThreads, 0, s>>>(p, in, out, n);
  return cudaGetLastError();
}
cudaError_t launch_ssd_init(const FieldView &f, float px, float py, float pz, float s1d, SSDState *st, SSDResult *res,
                            cudaStream_t s) {
  count_launch();
  ssd_init_kernel<<<1, 32, 0, s>>>(f, px, py, pz, s1d, st, res);
  return cudaGetLastError();
}
cudaError_t launch_ssd_cosine(SSDState *st, float nx, float ny, float nz, float ck, float cn, cudaStream_t s) {
  count_launch();
  ssd_cosine_kernel<<<1, 32, 0, s>>>(st, nx, ny, nz, ck, cn);
  return cudaGetLastError();
}
cudaError_t launch_ssd_hg(SSDState *st, float dx, float dy, float dz, float meanCosine, cudaStream_t s) {
  count_launch();
  ssd_hg_kernel<<<1, 32, 0, s>>>(st, dx, dy, dz, meanCosine);
  return cudaGetLastError();
}
cudaError_t launch_ssd_sample(const SSDState *st, float ux, float uy, int withPdf, SSDResult *res, cudaStream_t s) {
  count_launch();
  ssd_sample_kernel<<<1, 32, 0, s>>>(st, ux, uy, withPdf, res);
  return cudaGetLastError();
}
cudaError_t launch_ssd_pdf(const SSDState *st, float dx, float dy, float dz, int li, SSDResult *res, cudaStream_t s) {
  count_launch();
  ssd_pdf_kernel<<<1, 32, 0, s>>>(st, dx, dy, dz, li, res);
  return cudaGetLastError();
}

}  // namespace pgl

namespace pgl {
cudaError_t launch_ssd_dqt_sample(const FieldView &f, const SSDState *st, float ux, float uy, SSDResult *res,
                                  cudaStream_t s) {
  count_launch();
  ssd_dqt_sample_kernel<<<1, 1, 0, s>>>(f, st, ux, uy, res);
  return cudaGetLastError();
}
cudaError_t launch_ssd_dqt_pdf(const FieldView &f, const SSDState *st, float dx, float dy, float dz, SSDResult *res,
                               cudaStream_t s) {
  count_launch();
  ssd_dqt_pdf_kernel<<<1, 1, 0, s>>>(f, st, dx, dy, dz, res);
  return cudaGetLastError();
}
}  // namespace pgl
