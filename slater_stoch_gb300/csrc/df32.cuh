// df32.cuh -- two-float ("double-float") arithmetic: a value is the unevaluated sum h + l of two
// floats, about 48 significant bits, from error-free transformations (T. J. Dekker, Numer. Math.
// 18 (1971) 224; D. E. Knuth, TAOCP 2, 4.2.2).
//
// On GB300 the FP32 pipe issues 64 times as many lanes per clock as the FP64 pipe, so an operation
// of 4 to 12 FP32 instructions is 5 to 16 times faster than its FP64 counterpart.  Sums are not
// renormalised: the low part may grow to a few units in the last place of the operands' high
// parts, and the error stays about 2^-47 of the operands' magnitude.
#pragma once

// The arithmetic is plain IEEE FP32 with explicit fma, so it also compiles as host C++ (the host
// build of the tests, contraction off).
#ifdef __CUDACC__
#define SS_DF __device__ __forceinline__
#else
#include <cmath>
#define SS_DF inline
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
#endif

namespace ss {

#ifdef __CUDACC__
SS_DF float df_rsqrt_seed(float x) { return rsqrtf(x); }
#else
SS_DF float df_rsqrt_seed(float x) { return 1.0f / std::sqrt(x); }
#endif

struct alignas(8) df {
  float h, l;
};

SS_DF df df_from(double x) {
  const float h = (float)x;
  return df{h, (float)(x - (double)h)};
}
SS_DF double df_to(df a) { return (double)a.h + (double)a.l; }
SS_DF df df_neg(df a) { return df{-a.h, -a.l}; }
// exact for a power of two k
SS_DF df df_scale(df a, float k) { return df{__fmul_rn(a.h, k), __fmul_rn(a.l, k)}; }
SS_DF df df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return df{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
// |a| >= |b| or a == 0
SS_DF df df_fast_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return df{s, __fsub_rn(b, __fsub_rn(s, a))};
}
SS_DF df df_add(df a, df b) {
  const df s = df_two_sum(a.h, b.h);
  return df{s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
SS_DF df df_sub(df a, df b) { return df_add(a, df_neg(b)); }
// a - b of three floats each, to two-float accuracy however much of the leading parts cancels
SS_DF df df_sub3(float a0, float a1, float a2, float b0, float b1, float b2) {
  const df s = df_two_sum(a0, -b0), t = df_two_sum(a1, -b1), u = df_two_sum(s.h, t.h);
  return df{u.h, __fadd_rn(u.l, __fadd_rn(s.l, __fadd_rn(t.l, __fsub_rn(a2, b2))))};
}
SS_DF df df_mul(df a, df b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  return df{p, __fmaf_rn(a.l, b.h, e)};
}
SS_DF df df_mulf(df a, float b) {
  const float p = __fmul_rn(a.h, b);
  return df{p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p))};
}
SS_DF df df_fma(df a, df b, df c) { return df_add(df_mul(a, b), c); }
// c dominates the product
SS_DF df df_fma_fast(df a, df b, df c) {
  const df p = df_mul(a, b), s = df_fast_sum(c.h, p.h);
  return df{s.h, __fadd_rn(s.l, __fadd_rn(p.l, c.l))};
}
SS_DF df df_renorm(df a) { return df_fast_sum(a.h, a.l); }
// 1/sqrt(a): a float estimate corrected to the nearest float, then its residual 1 - a y^2
SS_DF df df_rsqrt(df a) {
  float y = df_rsqrt_seed(a.h);
  float r = 0.f;
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const float p = __fmul_rn(y, y);
    const float pe = __fmaf_rn(y, y, -p);
    r = __fmaf_rn(a.h, p, -1.f);
    r = __fmaf_rn(a.h, pe, r);
    r = __fmaf_rn(a.l, p, r);                              // a y^2 - 1
    r = __fmul_rn(r, __fmaf_rn(0.375f, r, -0.5f));         // (1 + r)^(-1/2) - 1
    if (it == 0) y = __fmaf_rn(y, r, y);
  }
  return df{y, __fmul_rn(y, r)};
}

}  // namespace ss
