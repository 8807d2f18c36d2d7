// Host build of the double-float exp and of the lobe normalisations
// (pgl_math.cuh), compiled with contraction off as the library: the largest
// relative error of the double-float exp against long double, how often the
// rounding tests give up, and decided results that differ from the double
// functions rounded once (which is what they stand for).
#include <cmath>
#include <cstdint>

#include "pgl_math.cuh"

using namespace pgl;

// every `stride`-th float of [begin, end) by bit pattern; out: inputs,
// undecided, wrong; *err: worst relative error
extern "C" void expf_df_check(uint32_t begin, uint32_t end, uint32_t stride, float margin, uint64_t *out, double *err) {
  for (uint64_t u = begin; u < end; u += stride) {
    const float x = u2f(uint32_t(u));
    ++out[0];
    if (fabsf(x) <= 87.0f) {
      int k;
      const DFloat m = exp_df_parts(x, &k);
      const long double e = ldexpl(expl((long double)x), -k);
      const double r = double(fabsl(((long double)m.h + (long double)m.l - e) / e));
      *err = r > *err ? r : *err;
    }
    float f;
    if (!expf_df(x, margin, &f)) ++out[1];
    else if (f2u(f) != f2u(float(std::exp(double(x))))) ++out[2];
  }
}
extern "C" void norms_df_check(const float *k, const float *e, const float *s, long n, uint64_t *out) {
  for (long i = 0; i < n; ++i) {
    float f;
    out[0] += 2;
    if (!vmf_norm_df(k[i], e[i], &f)) ++out[1];
    else if (f2u(f) != f2u(vmf_norm_double(k[i], e[i]))) ++out[2];
    if (!scale_norm_df(s[i], e[i], k[i] * k[i], &f)) ++out[1];
    else if (f2u(f) != f2u(scale_norm_double(s[i], e[i], k[i] * k[i]))) ++out[2];
  }
}
