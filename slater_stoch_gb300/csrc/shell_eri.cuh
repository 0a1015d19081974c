// shell_eri.cuh -- the shell-quartet ERI kernel (instantiated per total degree in shell_k*.cu).
//
// Replaces gauss_ijkl (src/gauss_ijkl.F90:51-154) for shells up to d and the r^2-type fits, by the
// scheme of McMurchie and Davidson (J. Comput. Phys. 26 (1978) 218): the product of two Gaussians
// is a sum of Hermite Gaussians with coefficients E, and the repulsion of two Hermite Gaussians is
// R_{t+tau}, a derivative of the Boys function.
//
// One CTA per (shell quartet, bra slice).  The (bra, ket) primitive items of the slice are
// numbered bra-major and taken in batches:
//  1. each thread forms the Hermite integrals of an item in registers and puts them in shared
//     memory (one row per item);
//  2. for each bra primitive of the batch, thread <-> (group, bra Hermite function, ket component)
//     sums R_{t+tau} E_tau over its group's items; when the bra primitive is done, its coefficients
//     contract the sums into the output block.
// Tiers: primitives are sorted by their Schwarz factor relative to the function pairs' diagonals
// (the largest over the components), so the kept kets of a bra primitive are a prefix, and those of
// each tier a range of it; each member of the shell quartet has at least the tier that it would
// have alone.  By the bound S_P S_Q of an item:
//   >= eps_df   FP64
//   >= eps32    two floats (df32.cuh, 48 bits): FP64 issues 2 lanes per clock and SM, FP32 128
//   >= eps      FP32
// Range of the FP32 exponent: over the primitives of a fit (2 alpha)^n spans more decades at n = 8
// than FP32 has.  An item's integrals are therefore formed in its own unit of length, R_n k^-n with
// k = min(s_P, s_Q) (about sqrt(2 alpha); powers of two, so scaling is exact), and the coefficients
// are E_t s^|t|.  What remains of a term is (k / s_P)^|t| (k / s_Q)^|tau|, at most one: where it
// underflows the term is negligible.  One unit for the whole shell quartet let the integrals of its
// diffuse primitives underflow: two centres and 30-Gaussian fits were wrong by 4e-7 of the Schwarz
// bound; the factors cost 2 to 6 % (26-function water 44.3 -> 46.1 ms).
// Centres are three floats: with two, the distance of two centres that nearly coincide kept 48 bits
// of their coordinates, and a molecule 120 bohr from the origin was wrong by up to 1e-10 of the bound;
// the third costs 0 to 3 % (46.1 -> 47.3 ms).  With both, the tiers differ from the all-FP64 evaluation
// by at most 2.3e-15 of the bound over the bases of tests/test_shell_range_gpu.py.
// The decomposition (slices, batches, groups) depends on the shell quartet alone, so a value does
// not depend on which other quartets were asked for.
#pragma once
#include <math.h>

#include <algorithm>
#include <utility>

#include "boys.cuh"
#include "df32.cuh"
#include "shell.cuh"

namespace ss {

#ifndef __CUDACC__  // the host build of the tests
using std::fma;
using std::min;
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
#endif

constexpr double SH_PI_5_2 = 34.9868366552;  // src/general_primitive_integral.F90:25

// F_0..F_L(T), T >= 0.  T <= 36: F_L from the Taylor series around T_k = k/8 (nine terms, |T - T_k|
// <= 1/16), then F_n = (2T F_{n+1} + e^-T) / (2n+1), stable; above, erf(sqrt T) = 1 and the upward
// recursion is stable.
template <int L>
SS_DF void boys_shell(double T, double (&F)[L + 1], const ShBoys* __restrict__ tab) {
  const int64_t tb = bits_of(T);
  if (tb <= 0x4042000000000000LL) {  // T <= 36
    const double t = fma(T, 8.0, RINT_SHIFT);
    // at most 288 for T <= 36; held there so that no value of T can index past the table
    const int k = (int)min((uint32_t)bits_of(t), (uint32_t)(SH_BOYS_K - 1));
    const double x = fma(t - RINT_SHIFT, 0.125, -T);  // T_k - T, exact
    const double* a = tab->a[k];
    double s = a[8];
#pragma unroll
    for (int j = 7; j >= 0; j--) s = fma(s, x, a[j]);
    F[L] = s;
    if (L > 0) {
      const double e = exp_neg(-T, exp2_32_tab), T2 = T + T;
#pragma unroll
      for (int n = L - 1; n >= 0; n--) F[n] = fma(T2, F[n + 1], e) * (1.0 / (2 * n + 1));
    }
  } else {
    const double u = rsqrt(T);
    F[0] = 0.88622692545275801365 * u;  // sqrt(pi)/2
    if (L > 0) {
      const double h = 0.5 * u * u;
      const double e = (tb > 0x4054000000000000LL) ? 0.0 : exp_neg(-T, exp2_32_tab);  // T > 80
#pragma unroll
      for (int n = 1; n <= L; n++) F[n] = fma((double)(2 * n - 1), F[n - 1], -e) * h;
    }
  }
}

// Two floats: the terms of degree >= 5 of the series in FP32 (they are below 1e-8 of F_L); above
// T = 36, e^-T is below 3e-16 and taken in FP32.
template <int L>
SS_DF void boys_shell(df T, df (&F)[L + 1], const float* tab) {
  if (T.h <= 36.f) {
    const int k = min((int)fmaf(T.h, 8.f, 0.5f), SH_BOYS_K - 1);
    const df x = df_fast_sum(__fsub_rn((float)k * 0.125f, T.h), -T.l);  // T_k - T
    const float4* row = reinterpret_cast<const float4*>(tab + k * SH_BOYS_ROW);
    const float4 r0 = row[0], r1 = row[1], r2 = row[2], r3 = row[3];
    float t = fmaf(r3.w, x.h, r3.z);
    t = fmaf(t, x.h, r3.y);
    t = fmaf(t, x.h, r3.x);
    df s = df_fast_sum(r2.x, __fmul_rn(t, x.h));
    s.l = __fadd_rn(s.l, r2.y);
    s = df_fma_fast(s, x, df{r1.z, r1.w});
    s = df_fma_fast(s, x, df{r1.x, r1.y});
    s = df_fma_fast(s, x, df{r0.z, r0.w});
    s = df_fma_fast(s, x, df{r0.x, r0.y});
    F[L] = s;
    if (L > 0) {
      // e^-T = e^-T_k e^x, |x| <= 1/16: degrees 5..9 in FP32
      float q = fmaf(x.h, 1.f / 362880, 1.f / 40320);
      q = fmaf(q, x.h, 1.f / 5040);
      q = fmaf(q, x.h, 1.f / 720);
      q = fmaf(q, x.h, 1.f / 120);
      df e = df_fast_sum(1.f / 24, __fmul_rn(q, x.h));
      e.l = __fadd_rn(e.l, (float)(1.0 / 24 - (double)(1.f / 24)));
      e = df_fma_fast(e, x, df{1.f / 6, (float)(1.0 / 6 - (double)(1.f / 6))});
      e = df_fma_fast(e, x, df{0.5f, 0.f});
      e = df_fma_fast(e, x, df{1.f, 0.f});
      e = df_fma_fast(e, x, df{1.f, 0.f});
      e = df_mul(e, df{r2.z, r2.w});
      const df T2 = df_scale(T, 2.f);
#pragma unroll
      for (int n = L - 1; n >= 0; n--) {
        const df v = df_fma(T2, F[n + 1], e);
        const float ih = 1.f / (2 * n + 1);
        F[n] = n == 0 ? v : df_mul(v, df{ih, (float)(1.0 / (2 * n + 1) - (double)ih)});
      }
    }
  } else {
    const df u = df_rsqrt(T);
    F[0] = df_mul(u, df{0.886226925f, (float)(0.88622692545275801365 - (double)0.886226925f)});
    if (L > 0) {
      const df h = df_scale(df_mul(u, u), 0.5f);
      const float e = T.h > 80.f ? 0.f : expf(-T.h);
#pragma unroll
      for (int n = 1; n <= L; n++) {
        df v = df_mulf(F[n - 1], (float)(2 * n - 1));
        v = df_fast_sum(v.h, __fsub_rn(v.l, e));
        F[n] = df_mul(v, h);
      }
    }
  }
}

// FP32, the same series to degree 5; above T = 30 the asymptotic F_0
template <int L>
SS_DF void boys_shell(float T, float (&F)[L + 1], const float* tab) {
  if (T >= 30.f) {
    const float h = 0.5f / T;
    const float e = expf(-T);
    F[0] = 0.886226925452758f * sqrtf(h + h);
#pragma unroll
    for (int n = 1; n <= L; n++) F[n] = fmaf((float)(2 * n - 1), F[n - 1], -e) * h;
    return;
  }
  const int k = (int)(T * 8.f + 0.5f);
  const float x = (float)k * 0.125f - T;
  const float* a = tab + k * SH_BOYS_ROW;
  float s = a[12];
#pragma unroll
  for (int j = 4; j >= 0; j--) s = fmaf(s, x, a[2 * j]);
  F[L] = s;
  if (L > 0) {
    const float e = expf(-T);
#pragma unroll
    for (int n = L - 1; n >= 0; n--) F[n] = fmaf(T + T, F[n + 1], e) * (1.f / (float)(2 * n + 1));
  }
}

// the operations of the recursion in each type
SS_DF double r_mul(double a, double b) { return a * b; }
SS_DF float r_mul(float a, float b) { return a * b; }
SS_DF df r_mul(df a, df b) { return df_mul(a, b); }
SS_DF double r_fma(double a, double b, double c) { return fma(a, b, c); }
SS_DF float r_fma(float a, float b, float c) { return fmaf(a, b, c); }
SS_DF df r_fma(df a, df b, df c) { return df_fma(a, b, c); }
SS_DF double r_times(double a, int n) { return n == 1 ? a : (double)n * a; }
SS_DF float r_times(float a, int n) { return n == 1 ? a : (float)n * a; }
SS_DF df r_times(df a, int n) {
  return n == 1 ? a : ((n & (n - 1)) == 0 ? df_scale(a, (float)n) : df_mulf(a, (float)n));
}

// (t, u, v) of a Hermite index
struct ShDeg {
  int t, u, v;
};
__host__ __device__ constexpr ShDeg sh_degs(int i) {
  int d = 0;
  while (sh_nherm(d) <= i) d++;
  const int r = d ? i - sh_nherm(d - 1) : 0;
  int w = 0;
  while ((w + 1) * (w + 2) / 2 <= r) w++;
  const int v = r - w * (w + 1) / 2;
  return ShDeg{d - w, w - v, v};
}

// One entry of the recursion below, all indices at compile time.
template <int I, typename Real, int N>
SS_DF void hermite_step(Real X, Real Y, Real Z, Real (&R)[N]) {
  constexpr ShDeg h = sh_degs(I);
  constexpr int big = 99;
  constexpr int at = h.t ? h.t : big, au = h.u ? h.u : big, av = h.v ? h.v : big;
  constexpr int ax = (at <= au && at <= av) ? 0 : (au <= av ? 1 : 2);
  constexpr int n = ax == 0 ? h.t : (ax == 1 ? h.u : h.v);
  constexpr int i1 = sh_hidx(h.t - (ax == 0), h.u - (ax == 1), h.v - (ax == 2));
  const Real x = ax == 0 ? X : (ax == 1 ? Y : Z);
  if constexpr (n == 1) {
    R[I] = r_mul(x, R[i1]);
  } else {
    constexpr int i2 = sh_hidx(h.t - 2 * (ax == 0), h.u - 2 * (ax == 1), h.v - 2 * (ax == 2));
    R[I] = r_fma(x, R[i1], r_times(R[i2], n - 1));
  }
}
template <typename Real, int N, int... I>
SS_DF void hermite_level(Real X, Real Y, Real Z, Real (&R)[N], std::integer_sequence<int, I...>) {
  (hermite_step<(int)sizeof...(I) - I>(X, Y, Z, R), ...);  // indices sizeof...(I) .. 1
}

// Hermite integrals of degree <= L in place: level m holds R^(m)_tuv, t + u + v <= L - m, and
// R^(m)_{t+1} = X R^(m+1)_t + t R^(m+1)_{t-1} (the axis with the smallest degree is lowered: a
// degree of one needs no second term).  Level m overwrites level m + 1 from the highest index
// down, so each entry reads values that are still of level m + 1.  base[m] = R^(m)_000.
template <int L, int M, typename Real>
SS_DF void hermite_levels(Real X, Real Y, Real Z, const Real (&base)[L + 1],
                                               Real (&R)[sh_nherm(L)]) {
  if constexpr (M >= 0) {
    hermite_level(X, Y, Z, R, std::make_integer_sequence<int, sh_nherm(L - M) - 1>());
    R[0] = base[M];
    hermite_levels<L, M - 1>(X, Y, Z, base, R);
  }
}

__host__ __device__ constexpr int sh_dfact(int n) { return n <= 1 ? 1 : n * sh_dfact(n - 2); }  // n!!

template <typename Real, int N, int... I>
SS_DF void put_row(const Real (&R)[N], Real* row, std::integer_sequence<int, I...>) {
  ((row[I] = R[I]), ...);
}
template <int L, typename Real>
SS_DF void store_row(Real X, Real Y, Real Z, const Real (&base)[L + 1], Real* row) {
  Real R[sh_nherm(L)];
  R[0] = base[L];
  hermite_levels<L, L - 1>(X, Y, Z, base, R);
  put_row(R, row, std::make_integer_sequence<int, sh_nherm(L)>());
}

// all four shells on one centre: only the even degrees, R_{2a 2b 2c} = (2a-1)!! (2b-1)!! (2c-1)!! base[a+b+c]
template <int I, typename Real, int N>
SS_DF void put_1c(const Real (&base)[N], Real* row) {
  constexpr ShDeg h = sh_degs(I);
  if constexpr (!((h.t | h.u | h.v) & 1)) {
    constexpr int c = sh_dfact(h.t - 1) * sh_dfact(h.u - 1) * sh_dfact(h.v - 1);
    row[I] = r_times(base[(h.t + h.u + h.v) / 2], c);
  }
}
template <typename Real, int N, int... I>
SS_DF void put_row_1c(const Real (&base)[N], Real* row, std::integer_sequence<int, I...>) {
  (put_1c<I>(base, row), ...);
}
template <int L, typename Real>
SS_DF void store_row_1c(const Real (&base)[L + 1], Real* row) {
  put_row_1c(base, row, std::make_integer_sequence<int, sh_nherm(L)>());
}

#ifdef __CUDACC__
__constant__ uint32_t sh_hermite[SH_MAXH] = {
#define H_(t, u, v) ((t) | ((u) << 8) | ((v) << 16))
    H_(0, 0, 0), H_(1, 0, 0), H_(0, 1, 0), H_(0, 0, 1), H_(2, 0, 0), H_(1, 1, 0), H_(1, 0, 1), H_(0, 2, 0),
    H_(0, 1, 1), H_(0, 0, 2), H_(3, 0, 0), H_(2, 1, 0), H_(2, 0, 1), H_(1, 2, 0), H_(1, 1, 1), H_(1, 0, 2),
    H_(0, 3, 0), H_(0, 2, 1), H_(0, 1, 2), H_(0, 0, 3), H_(4, 0, 0), H_(3, 1, 0), H_(3, 0, 1), H_(2, 2, 0),
    H_(2, 1, 1), H_(2, 0, 2), H_(1, 3, 0), H_(1, 2, 1), H_(1, 1, 2), H_(1, 0, 3), H_(0, 4, 0), H_(0, 3, 1),
    H_(0, 2, 2), H_(0, 1, 3), H_(0, 0, 4)
#undef H_
};
__device__ __forceinline__ int sh_degree(uint32_t h) { return (int)((h & 255) + ((h >> 8) & 255) + (h >> 16)); }

__device__ __forceinline__ df sh_distance(const ShPrimF& a, const ShPrimF& b, int ax) {
  return df_sub3(a.ph[ax], a.pl[ax], a.pm[ax], b.ph[ax], b.pl[ax], b.pm[ax]);
}

// (k / s_Q)^dtau (k / s_P)^dt of an item, k = min(s_P, s_Q), from the exponents of s_Q / k and s_P / k as
// float bits (one of them is zero; both below 32, so the factor is a normal number)
__device__ __forceinline__ int2 sh_shift(const ShPrimF& a, const ShPrimF& b) {
  const int d = __float_as_int(b.s) - __float_as_int(a.s);
  return make_int2(min(max(d, 0), 31 << 23), min(max(-d, 0), 31 << 23));
}
__device__ __forceinline__ float sh_factor(int2 sh, int dtau, int dt) {
  return __int_as_float(0x3f800000 - sh.x * dtau - sh.y * dt);
}

// Threads of a CTA and items of a batch: rows of 8 bytes x Hermite integrals bound the batch from
// degree 5 on, where the sums of step 2 are most of the work.
template <int L>
struct ShDim {
  static constexpr int NT = L >= 6 ? 256 : 128;
  static constexpr int NB = L >= 5 ? 64 : 128;
  static constexpr int MINB = L >= 6 ? 2 : 4;  // CTAs per SM the registers must allow
  static constexpr int ROW = sh_nherm(L) | 1;  // odd: a column over the items meets no bank twice
  static_assert(NB % 2 == 0, "the columns after the rows begin on 16 bytes");
  // max_col: a multiple of 16
  static size_t bytes(int max_no, int max_ni, int max_col) {
    return sizeof(float) * SH_BOYS_K * SH_BOYS_ROW +
           sizeof(double) * ((size_t)NB * ROW + (max_no > NT ? max_no : NT) + max_ni) + (size_t)max_col;
  }
};

template <int L>
__global__ void __launch_bounds__(ShDim<L>::NT, ShDim<L>::MINB) shell_eri_kernel(ShArgs A, int max_no, int max_ni, int max_col) {
  constexpr int NT = ShDim<L>::NT, NB = ShDim<L>::NB, ROW = ShDim<L>::ROW;
  extern __shared__ float4 sh_raw[];
  float* s_boys = reinterpret_cast<float*>(sh_raw);                          // [SH_BOYS_K][SH_BOYS_ROW]
  double* s_R = reinterpret_cast<double*>(s_boys + SH_BOYS_K * SH_BOYS_ROW);  // [NB][ROW]: double, df or float
  uint8_t* s_col = reinterpret_cast<uint8_t*>(s_R + (size_t)NB * ROW);  // [ket term][bra Hermite]: column of t + tau
  double* s_acc = reinterpret_cast<double*>(s_col + max_col);  // [group][bra Hermite][ket component]: double or df
  double* s_out = s_acc + (max_no > NT ? max_no : NT);
  __shared__ int s_scan[3][SH_MAXSLICE + 1], s_first[3][SH_MAXSLICE], s_p[SH_MAXSLICE];
  __shared__ int2 s_sh[NB];  // exponents (as float bits) of s_Q / k and s_P / k of an item
  const int tid = threadIdx.x;
  {  // the launch's dynamic shared memory must hold this carve-up: checked, not assumed
    uint32_t dyn;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if (reinterpret_cast<char*>(s_out + max_ni) - reinterpret_cast<char*>(sh_raw) > (ptrdiff_t)dyn) return;
  }

  const ShWork W = A.work[A.cta[A.cta0 + blockIdx.x]];
  const int slice = A.cta0 + (int)blockIdx.x - W.cta0;
  const ShPair B = A.pair[W.bra], K = A.pair[W.ket];
  const int nb = A.cnt[W.bra], nk = A.cnt[W.ket];
  const ShPrim* bra = A.prim + B.prim_off;
  const ShPrim* ket = A.prim + K.prim_off;
  const ShStruct& SB = A.st[B.st];
  const ShStruct& SK = A.st[K.st];
  const ShBoys* boys = A.boys + L;
  const bool diag = A.diag != 0;
  const bool onec = B.onec && K.onec && bra[0].P[0] == ket[0].P[0] && bra[0].P[1] == ket[0].P[1] &&
                    bra[0].P[2] == ket[0].P[2];
  const int H = sh_nherm(B.d), nf = K.ncomp, NO = H * nf, NI = B.ncomp * nf, nterm = K.nterm;
  const uint64_t mask = W.mask;
  if (NO > (max_no > NT ? max_no : NT) || NI > max_ni || sh_col_size(B.d, nterm) > max_col || B.d + K.d != L) return;  // uniform

  // the tiers below FP64 of a quartet with a lane kernel are that kernel's
  const int tiers = diag || W.lane >= 0 ? 1 : 3;
  const int64_t stride = W.split + W.lsplit;
  if (tiers > 1) {
    const float4* src = reinterpret_cast<const float4*>(boys->f);
    for (int i = tid; i < SH_BOYS_K * SH_BOYS_ROW / 4; i += NT) sh_raw[i] = src[i];
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(A.col + K.col[B.d]);
    uint4* dst = reinterpret_cast<uint4*>(s_col);
    for (int i = tid; i < sh_col_size(B.d, nterm) / 16; i += NT) dst[i] = src[i];
  }
  for (int i = tid; i < NI; i += NT) s_out[i] = 0.0;

  // the slice's bra primitives (slice, slice + split, ...) and their ket ranges
  int ns = 0;
  if (slice < nb) ns = min(SH_MAXSLICE, (nb - slice + W.split - 1) / W.split);
  if (tid < SH_MAXSLICE) {
    const int p = slice + tid * W.split;
    int c = 0, cd = 0, cf = 0;  // ranges [0, cd) FP64, [cd, cf) two floats, [cf, c) FP32
    if (tid < ns) {
      c = cd = cf = diag ? p + 1 : nk;
      if (!diag) {
        const double sb = bra[p].S;
        auto first_below = [&](double thr) {  // first ket with sb * S < thr
          int lo = 0, hi = nk;
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sb * ket[mid].S < thr) hi = mid; else lo = mid + 1;
          }
          return lo;
        };
        c = first_below(A.eps);
        cd = cf = c;
        if (A.eps32 > A.eps) {
          cf = first_below(A.eps32);
          cd = first_below(A.eps_df);
        }
      }
      s_p[tid] = p;
    }
    s_first[0][tid] = 0;
    s_first[1][tid] = cd;
    s_first[2][tid] = cf;
    s_scan[0][tid + 1] = cd;
    s_scan[1][tid + 1] = cf - cd;
    s_scan[2][tid + 1] = c - cf;
  }
  __syncthreads();
  if (tid < 3) {
    s_scan[tid][0] = 0;
    for (int j = 0; j < SH_MAXSLICE; j++) s_scan[tid][j + 1] += s_scan[tid][j];
  }
  // this thread's place in step 2 when a bra primitive's sums fit the CTA
  const int G = NO < NT ? NT / NO : 1;
  const int my_g = NO < NT ? tid / NO : 0;
  const int my_o = NO < NT ? tid - my_g * NO : tid;
  for (int o = tid; o < (NO > NT ? NO : NT); o += NT) s_acc[o] = 0.0;
  const double scale = diag ? 1.0 : A.scale[W.bra] * A.scale[W.ket];
  __syncthreads();

  for (int tier = 0; tier < tiers; tier++) {
    const int* scan = s_scan[tier];
    const int n = scan[SH_MAXSLICE];
    for (int base = 0; base < n; base += NB) {
      const int top = min(base + NB, n);
      // ---- 1. one item per thread ----
      for (int item = base + tid; item < top; item += NT) {
        int j = 0;
#pragma unroll
        for (int s = SH_MAXSLICE / 2; s > 0; s >>= 1)
          if (scan[j + s] <= item) j += s;
        const int p = s_p[j];
        const int q = item - scan[j] + s_first[tier][j];
        if (tier == 0) {
          double* row = s_R + (item - base) * ROW;
          const ShPrim a = bra[p], b = ket[q];
          double pre = a.w * b.w;
          if (diag && q < p) pre = pre + pre;
          const double rs = rsqrt(a.p + b.p);
          pre *= rs;
          const double alpha = a.p * b.p * (rs * rs);
          const double m2a = -2.0 * alpha;
          double bs[L + 1];
          if (onec) {
            bs[0] = pre;
            double pw = pre;
#pragma unroll
            for (int m = 1; m <= L; m++) {
              pw *= m2a;
              bs[m] = pw * (1.0 / (2 * m + 1));
            }
            store_row_1c<L, double>(bs, row);
          } else {
            const double X = a.P[0] - b.P[0], Y = a.P[1] - b.P[1], Z = a.P[2] - b.P[2];
            double F[L + 1];
            boys_shell<L>(alpha * fma(X, X, fma(Y, Y, Z * Z)), F, boys);
            double pw = pre;
#pragma unroll
            for (int m = 0; m <= L; m++) {
              bs[m] = pw * F[m];
              if (m < L) pw *= m2a;
            }
            store_row<L, double>(X, Y, Z, bs, row);
          }
          continue;
        }
        const ShPrimF a = A.primf[B.prim_off + p], b = A.primf[K.prim_off + q];
        const float kx = fminf(a.s, b.s), ik = fmaxf(a.is, b.is), ik2 = ik * ik;
        s_sh[item - base] = sh_shift(a, b);
        if (tier == 1) {
          df* row = reinterpret_cast<df*>(s_R) + (item - base) * ROW;
          const df pa{a.p[0], a.p[1]}, pb{b.p[0], b.p[1]};
          const df rs = df_rsqrt(df_add(pa, pb));
          const df pre = df_mul(df_mul(df{a.w[0], a.w[1]}, df{b.w[0], b.w[1]}), rs);
          const df alpha = df_mul(df_mul(pa, rs), df_mul(pb, rs));
          const df m2a = df_scale(alpha, -2.f * ik2);
          df bs[L + 1];
          if (onec) {
            bs[0] = pre;
            df pw = pre;
#pragma unroll
            for (int m = 1; m <= L; m++) {
              const float ih = 1.f / (2 * m + 1);
              pw = df_mul(pw, m2a);
              bs[m] = df_mul(pw, df{ih, (float)(1.0 / (2 * m + 1) - (double)ih)});
            }
            store_row_1c<L, df>(bs, row);
          } else {
            const df X = sh_distance(a, b, 0), Y = sh_distance(a, b, 1), Z = sh_distance(a, b, 2);
            df F[L + 1];
            boys_shell<L>(df_renorm(df_mul(alpha, df_fma(X, X, df_fma(Y, Y, df_mul(Z, Z))))), F, s_boys);
            df pw = pre;
#pragma unroll
            for (int m = 0; m <= L; m++) {
              bs[m] = df_mul(pw, F[m]);
              if (m < L) pw = df_mul(pw, m2a);
            }
            store_row<L, df>(df_scale(X, kx), df_scale(Y, kx), df_scale(Z, kx), bs, row);
          }
        } else {
          float* row = reinterpret_cast<float*>(s_R) + (item - base) * ROW;
          float pre = a.w[0] * b.w[0];
          const float rs = rsqrtf(a.p[0] + b.p[0]);
          pre *= rs;
          const float alpha = (a.p[0] * rs) * (b.p[0] * rs);
          const float m2a = -2.f * (alpha * ik2);
          float bs[L + 1];
          if (onec) {
            bs[0] = pre;
            float pw = pre;
#pragma unroll
            for (int m = 1; m <= L; m++) {
              pw *= m2a;
              bs[m] = pw * (1.f / (2 * m + 1));
            }
            store_row_1c<L, float>(bs, row);
          } else {
            const float X = (a.ph[0] - b.ph[0]) + (a.pl[0] - b.pl[0]);
            const float Y = (a.ph[1] - b.ph[1]) + (a.pl[1] - b.pl[1]);
            const float Z = (a.ph[2] - b.ph[2]) + (a.pl[2] - b.pl[2]);
            float F[L + 1];
            boys_shell<L>(alpha * fmaf(X, X, fmaf(Y, Y, Z * Z)), F, s_boys);
            float pw = pre;
#pragma unroll
            for (int m = 0; m <= L; m++) {
              bs[m] = pw * F[m];
              if (m < L) pw *= m2a;
            }
            store_row<L, float>(X * kx, Y * kx, Z * kx, bs, row);
          }
        }
      }
      __syncthreads();
      // ---- 2. segments of the batch: runs of one bra primitive ----
      int j = 0;
#pragma unroll
      for (int s = SH_MAXSLICE / 2; s > 0; s >>= 1)
        if (scan[j + s] <= base) j += s;
      int lo = base;
      while (lo < top) {
        while (scan[j + 1] <= lo) j++;
        // with an s-type bra the FP64 sums need no contraction and no segments
        const int hi = (H == 1 && tier == 0) ? top : min(top, scan[j + 1]);
        const int i0 = lo - base + my_g, i1 = hi - base;
        const int q0 = lo - scan[j] + s_first[tier][j] + my_g;  // ket of the thread's first item
        for (int o = my_o; o < NO && my_g < G; o += NT) {
          const int t = o / nf, f = o - t * nf;
          if ((mask >> f) & 1) {
            const uint32_t ht = sh_hermite[t];
            const int x1 = SK.fs[f + 1];
            if (tier == 0) {
              double acc = 0.0;
              for (int x = SK.fs[f]; x < x1; x++) {
                const uint32_t tau = SK.term[x];
                if (onec && ((ht + tau) & 0x010101u)) continue;  // odd degrees vanish on one centre
                const double* Rc = s_R + s_col[x * H + t];
                double s = 0.0;
                if (H == 1) {  // items of several bra primitives: the kets are not consecutive
                  int jj = j;
                  for (int i = i0; i < i1; i += G) {
                    while (scan[jj + 1] <= base + i) jj++;
                    const int q = base + i - scan[jj] + s_first[0][jj];
                    s = fma(Rc[i * ROW], A.E[K.e_off + (size_t)q * nterm + x], s);
                  }
                } else {
                  const double* Ek = A.E + K.e_off + (size_t)q0 * nterm + x;
#pragma unroll 4
                  for (int i = i0; i < i1; i += G, Ek += (size_t)G * nterm) s = fma(Rc[i * ROW], *Ek, s);
                }
                acc += (sh_degree(tau) & 1) ? -s : s;
              }
              s_acc[o + my_g * NO] += acc;
            } else {
              df acc = reinterpret_cast<df*>(s_acc)[o + my_g * NO];
              for (int x = SK.fs[f]; x < x1; x++) {
                const uint32_t tau = SK.term[x];
                if (onec && ((ht + tau) & 0x010101u)) continue;
                const float2* Ek = A.E2 + K.e_off + (size_t)q0 * nterm + x;
                const int col = s_col[x * H + t];
                const int dtau = sh_degree(tau), dt = sh_degree(ht);
                const float sign = (dtau & 1) ? -1.f : 1.f;
                if (tier == 1) {
                  const df* Rc = reinterpret_cast<const df*>(s_R) + col;
                  df s{0.f, 0.f};
#pragma unroll 4
                  for (int i = i0; i < i1; i += G, Ek += (size_t)G * nterm) {
                    const float2 e = *Ek;
                    s = df_fma(Rc[i * ROW], df_scale(df{e.x, e.y}, sh_factor(s_sh[i], dtau, dt)), s);
                  }
                  acc = df_add(acc, df_scale(s, sign));
                } else {
                  const float* Rc = reinterpret_cast<const float*>(s_R) + col;
                  float s = 0.f;
#pragma unroll 4
                  for (int i = i0; i < i1; i += G, Ek += (size_t)G * nterm)
                    s = fmaf(Rc[i * ROW], Ek->x * sh_factor(s_sh[i], dtau, dt), s);
                  acc = df_add(acc, df{s * sign, 0.f});
                }
              }
              reinterpret_cast<df*>(s_acc)[o + my_g * NO] = df_renorm(acc);
            }
          }
          if (NO < NT) break;
        }
        const bool done = H == 1 ? (base + NB >= n && hi == top) : hi == scan[j + 1];
        if (done) {  // the sums of this bra primitive (s-type bra: of the tier) are complete
          __syncthreads();
          for (int o = tid; o < NO; o += NT) {
            double v;
            if (tier == 0) {
              v = s_acc[o];
              for (int g = 1; g < G; g++) v += s_acc[o + g * NO];
            } else {
              const df* acc = reinterpret_cast<const df*>(s_acc);
              df sum = acc[o];
              for (int g = 1; g < G; g++) sum = df_add(sum, acc[o + g * NO]);
              v = df_to(sum) * scale;
              // the sums are in the bra primitive's unit (degree 0 where they hold several primitives')
              if (H > 1)
                for (int d = sh_degree(sh_hermite[o / nf]); d > 0; d--) v *= (double)A.primf[B.prim_off + s_p[j]].s;
            }
            for (int g = 1; g < G; g++) s_acc[o + g * NO] = 0.0;
            s_acc[o] = v;
          }
          __syncthreads();
          const double* Eb = A.E + B.e_off + (size_t)s_p[H == 1 ? 0 : j] * B.nterm;
          for (int e = tid; e < NI; e += NT) {
            const int a = e / nf, f = e - a * nf;
            if (!((mask >> f) & 1) || (diag && a != f)) continue;
            double s = 0.0;
            for (int x = SB.fs[a]; x < SB.fs[a + 1]; x++) s = fma(Eb[x], s_acc[sh_pack_idx(SB.term[x]) * nf + f], s);
            s_out[e] += s;
          }
          __syncthreads();
          for (int o = tid; o < NO; o += NT) s_acc[o] = 0.0;
        }
        lo = hi;
      }
      __syncthreads();
    }
  }
  if (diag) {
    for (int a = tid; a < nf; a += NT) A.partial[W.part + a * stride + slice] = SH_PI_5_2 * s_out[a * nf + a];
  } else {
    for (int e = tid; e < NI; e += NT) A.partial[W.part + e * stride + slice] = SH_PI_5_2 * s_out[e];
  }
}

template <int L>
cudaError_t launch_shell_L(int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A) {
  const size_t smem = ShDim<L>::bytes(max_no, max_ni, max_col);
  if (smem > SH_SMEM_MAX) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(shell_eri_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, SH_SMEM_MAX);
  if (e != cudaSuccess) return e;
  shell_eri_kernel<L><<<ncta, ShDim<L>::NT, smem, st>>>(A, max_no, max_ni, max_col);
  return cudaGetLastError();
}

#endif  // __CUDACC__

}  // namespace ss
