// shell_eri.cuh -- the shell-quartet ERI kernel (instantiated per total degree in shell_k*.cu).
//
// Replaces gauss_ijkl (src/gauss_ijkl.F90:51-154) for shells up to d and the r^2-type fits, by the
// scheme of McMurchie and Davidson (J. Comput. Phys. 26 (1978) 218): the product of two Gaussians
// is a sum of Hermite Gaussians with coefficients E, and the repulsion of two Hermite Gaussians is
// R_{t+tau}, a derivative of the Boys function.
//
// What bounds it: the FP64 pipe (2 fused multiply-adds per clock and SM).  A warp's FP64
// instruction occupies it for 16 clocks, so shared-memory operands and index arithmetic are free
// and only the number of FP64 operations counts.  Per primitive quartet of four shells it takes
// one Boys evaluation, the Hermite recursion, and one multiply-add per (bra Hermite function, ket
// Hermite coefficient); the bra's coefficients are applied once per bra primitive, after the sum
// over the ket's.
//
// One CTA per (shell quartet, bra slice).  The (bra, ket) primitive items of the slice are
// numbered bra-major and taken in batches of one item per thread:
//  1. each thread forms the Hermite integrals of its item in registers and puts them in shared
//     memory (one row per item);
//  2. for each bra primitive of the batch, thread <-> (group, bra Hermite function, ket component)
//     sums R_{t+tau} E_tau over its group's items; when the bra primitive is done, its coefficients
//     contract the sums into the output block.
// Tiers as in eri_kernel.cuh: primitives are sorted by their Schwarz factor relative to the
// function pairs' diagonals (the largest over the components), so the kept kets of a bra
// primitive are a prefix, and those evaluated in FP64 a shorter one; each member of the shell
// quartet therefore has at least the tier that it would have alone.
// The decomposition (slices, batches, groups) depends on the shell quartet alone, so a value does
// not depend on which other quartets were asked for.
#pragma once
#include <math.h>

#include "boys.cuh"
#include "boys_grid.cuh"
#include "shell.cuh"

namespace ss {

constexpr double SH_PI_5_2 = 34.9868366552;  // src/general_primitive_integral.F90:25
constexpr int SH_MAXSLICE = 16;              // bra primitives of a slice

// F_0..F_L(T), T >= 0.  T <= 36: F_L from the Taylor series around T_k = k/8 (row k of tab: F_{L+j}(T_k) / j!,
// j < 9), then F_n = (2T F_{n+1} + e^-T) / (2n+1), stable; above, erf(sqrt T) = 1 and the upward
// recursion is stable.
template <int L>
__device__ __forceinline__ void boys_shell(double T, double (&F)[L + 1], const double* tab, const double* e2) {
  const int64_t tb = bits_of(T);
  if (tb <= 0x4042000000000000LL) {  // T <= 36
    const double t = fma(T, 8.0, RINT_SHIFT);
    // at most 288 for T <= 36; held there so that no value of T can index past the table
    const int k = (int)min((uint32_t)bits_of(t), (uint32_t)(BOYS_GRID_K - 1));
    const double x = fma(t - RINT_SHIFT, 0.125, -T);  // T_k - T, exact
    const double* a = tab + k * 9;
    double s = a[8];
#pragma unroll
    for (int j = 7; j >= 0; j--) s = fma(s, x, a[j]);
    F[L] = s;
    if (L > 0) {
      const double e = exp_neg(-T, e2), T2 = T + T;
#pragma unroll
      for (int n = L - 1; n >= 0; n--) F[n] = fma(T2, F[n + 1], e) * (1.0 / (2 * n + 1));
    }
  } else {
    const double u = rsqrt(T);
    F[0] = 0.88622692545275801365 * u;  // sqrt(pi)/2
    if (L > 0) {
      const double h = 0.5 * u * u;
      const double e = (tb > 0x4054000000000000LL) ? 0.0 : exp_neg(-T, e2);  // T > 80
#pragma unroll
      for (int n = 1; n <= L; n++) F[n] = fma((double)(2 * n - 1), F[n - 1], -e) * h;
    }
  }
}

// FP32: as boys32 (boys.cuh), table columns F_{L+j}(T_k) / j!, j < 6
template <int L>
__device__ __forceinline__ void boys_shell(float T, float (&F)[L + 1], const float* tab) {
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
  const float* a = tab + k * 6;
  float s = a[5];
#pragma unroll
  for (int j = 4; j >= 0; j--) s = fmaf(s, x, a[j]);
  F[L] = s;
  if (L > 0) {
    const float e = expf(-T);
#pragma unroll
    for (int n = L - 1; n >= 0; n--) F[n] = fmaf(T + T, F[n + 1], e) * (1.f / (float)(2 * n + 1));
  }
}

// Hermite integrals of degree <= L in place: level m holds R^(m)_tuv, t + u + v <= L - m, and
// R^(m)_{t+1} = X R^(m+1)_t + t R^(m+1)_{t-1} (the axis with the smallest degree is lowered: a
// degree of one needs no second term).  Level m overwrites level m + 1 from the highest degree
// down, so each entry reads values that are still of level m + 1.  base[m] = R^(m)_000.
template <int L, typename Real>
__device__ __forceinline__ void hermite_recursion(Real X, Real Y, Real Z, const Real (&base)[L + 1],
                                                  Real (&R)[sh_nherm(L)]) {
  R[0] = base[L];
#pragma unroll
  for (int mm = 0; mm < L; mm++) {  // level m = L - 1 - mm
#pragma unroll
    for (int dd = 0; dd <= mm; dd++) {
      const int d = mm + 1 - dd;
#pragma unroll
      for (int w = 0; w <= d; w++)
#pragma unroll
        for (int v = 0; v <= w; v++) {
          const int t = d - w, u = w - v;
          const int big = 99;
          const int at = t ? t : big, au = u ? u : big, av = v ? v : big;
          const int ax = (at <= au && at <= av) ? 0 : (au <= av ? 1 : 2);
          const int n = ax == 0 ? t : (ax == 1 ? u : v);
          const Real x = ax == 0 ? X : (ax == 1 ? Y : Z);
          const int i1 = sh_hidx(t - (ax == 0), u - (ax == 1), v - (ax == 2));
          if (n == 1) {
            R[sh_hidx(t, u, v)] = x * R[i1];
          } else {
            const int i2 = sh_hidx(t - 2 * (ax == 0), u - 2 * (ax == 1), v - 2 * (ax == 2));
            const Real b = n == 2 ? R[i2] : (Real)(n - 1) * R[i2];
            R[sh_hidx(t, u, v)] = fma(x, R[i1], b);
          }
        }
    }
    R[0] = base[L - 1 - mm];
  }
}

__host__ __device__ constexpr int sh_dfact(int n) { return n <= 1 ? 1 : n * sh_dfact(n - 2); }  // n!!

template <int L, typename Real>
__device__ __forceinline__ void store_row(Real X, Real Y, Real Z, const Real (&base)[L + 1], Real* row) {
  Real R[sh_nherm(L)];
  hermite_recursion<L, Real>(X, Y, Z, base, R);
#pragma unroll
  for (int i = 0; i < sh_nherm(L); i++) row[i] = R[i];
}

// all four shells on one centre: only the even degrees, R_{2a 2b 2c} = (2a-1)!! (2b-1)!! (2c-1)!! base[a+b+c]
template <int L, typename Real>
__device__ __forceinline__ void store_row_1c(const Real (&base)[L + 1], Real* row) {
#pragma unroll
  for (int a = 0; 2 * a <= L; a++)
#pragma unroll
    for (int b = 0; 2 * (a + b) <= L; b++)
#pragma unroll
      for (int c = 0; 2 * (a + b + c) <= L; c++)
        row[sh_hidx(2 * a, 2 * b, 2 * c)] =
            base[(a + b + c) % (L + 1)] * (Real)(sh_dfact(2 * a - 1) * sh_dfact(2 * b - 1) * sh_dfact(2 * c - 1));
}

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

template <int L>
struct ShSmem {
  static constexpr int NT = sh_threads(L);
  static constexpr int ROW = sh_row(L);
  static size_t bytes(int max_no, int max_ni) {
    return sizeof(double) * (BOYS_GRID_K * 9 + 32 + (size_t)NT * ROW + (max_no > NT ? max_no : NT) + max_ni) +
           sizeof(float) * BOYS32_K * 6 + sizeof(int) * NT;
  }
};

template <int L>
__global__ void __launch_bounds__(sh_threads(L)) shell_eri_kernel(ShArgs A, int max_no, int max_ni) {
  constexpr int NT = ShSmem<L>::NT;
  constexpr int ROW = ShSmem<L>::ROW;
  extern __shared__ double sh_raw[];
  double* s_boys = sh_raw;                       // [BOYS_GRID_K][9]
  double* s_e2 = s_boys + BOYS_GRID_K * 9;       // [32]
  double* s_R = s_e2 + 32;                       // [NT][ROW] (float rows in the FP32 pass)
  double* s_acc = s_R + (size_t)NT * ROW;        // [groups][bra Hermite][ket component]
  double* s_out = s_acc + (max_no > NT ? max_no : NT);
  float* s_boys32 = reinterpret_cast<float*>(s_out + max_ni);  // [BOYS32_K][6]
  int* s_q = reinterpret_cast<int*>(s_boys32 + BOYS32_K * 6);  // ket primitive of each item
  __shared__ int s_scan[2][SH_MAXSLICE + 1], s_c64[SH_MAXSLICE], s_p[SH_MAXSLICE];
  const int tid = threadIdx.x;
  {  // the launch's dynamic shared memory must hold this carve-up: checked, not assumed
    uint32_t dyn;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if (reinterpret_cast<char*>(s_q + NT) - reinterpret_cast<char*>(sh_raw) > (ptrdiff_t)dyn) return;  // block-uniform
  }

  const ShWork W = A.work[A.cta[A.cta0 + blockIdx.x]];
  const int slice = A.cta0 + (int)blockIdx.x - W.cta0;
  const ShPair B = A.pair[W.bra], K = A.pair[W.ket];
  const int nb = A.cnt[W.bra], nk = A.cnt[W.ket];
  const ShPrim* bra = A.prim + B.prim_off;
  const ShPrim* ket = A.prim + K.prim_off;
  const ShStruct& SB = A.st[B.st];
  const ShStruct& SK = A.st[K.st];
  const bool diag = A.diag != 0;
  const bool onec = B.onec && K.onec && bra[0].P[0] == ket[0].P[0] && bra[0].P[1] == ket[0].P[1] &&
                    bra[0].P[2] == ket[0].P[2];
  const int H = sh_nherm(B.d), nf = K.ncomp, NO = H * nf, NI = B.ncomp * nf;
  const uint64_t mask = W.mask;
  if (NO > (max_no > NT ? max_no : NT) || NI > max_ni || B.d + K.d != L) return;  // block-uniform

  for (int i = tid; i < BOYS_GRID_K * 9; i += NT) {
    const int k = i / 9, j = i - 9 * k;
    double f = boys_grid_tab[k * BOYS_GRID_N + L + j];
    const double inv[9] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320};
    double s = 1.0;
#pragma unroll
    for (int t = 0; t < 9; t++) s = j == t ? inv[t] : s;
    s_boys[i] = f * s;
  }
  for (int i = tid; i < 32; i += NT) s_e2[i] = exp2_32_tab[i];
  for (int i = tid; i < BOYS32_K * 6; i += NT) {
    const int k = i / 6, j = i - 6 * k;
    const float inv[6] = {1.f, 1.f, 0.5f, 1.f / 6, 1.f / 24, 1.f / 120};
    float s = 1.f;
#pragma unroll
    for (int t = 0; t < 6; t++) s = j == t ? inv[t] : s;
    s_boys32[i] = boys32_tab[k * BOYS32_N + L + j] * s;
  }
  for (int i = tid; i < NI; i += NT) s_out[i] = 0.0;

  // the slice's bra primitives (slice, slice + split, ...) and their ket prefixes
  int ns = 0;
  if (slice < nb) ns = min(SH_MAXSLICE, (nb - slice + W.split - 1) / W.split);
  if (tid < SH_MAXSLICE) {
    const int p = slice + tid * W.split;
    int c = 0, c64 = 0;
    if (tid < ns) {
      c = c64 = diag ? p + 1 : nk;
      if (!diag && A.eps > 0.0) {
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
        c64 = A.eps32 > A.eps ? first_below(A.eps32) : c;
      }
      s_p[tid] = p;
    }
    s_c64[tid] = c64;
    s_scan[0][tid + 1] = c64;
    s_scan[1][tid + 1] = c - c64;
  }
  __syncthreads();
  if (tid < 2) {
    s_scan[tid][0] = 0;
    for (int j = 0; j < SH_MAXSLICE; j++) s_scan[tid][j + 1] += s_scan[tid][j];
  }
  // this thread's place in step 2 when a segment's outputs fit the CTA
  const int G = NO < NT ? NT / NO : 1;
  const int my_g = NO < NT ? tid / NO : 0;
  const int my_o = NO < NT ? tid - my_g * NO : tid;
  for (int o = tid; o < (NO > NT ? NO : NT); o += NT) s_acc[o] = 0.0;
  __syncthreads();

  // sums of the bra primitive in slot j are complete: contract with its coefficients
  auto flush = [&](int j, float kx) {
    __syncthreads();
    for (int o = tid; o < NO; o += NT) {
      double v = s_acc[o];
      for (int g = 1; g < G; g++) {
        v += s_acc[o + g * NO];
        s_acc[o + g * NO] = 0.0;
      }
      if (kx != 1.f) {  // undo the FP32 pass's degree scaling (powers of two: exact)
        for (int d = sh_degree(sh_hermite[o / nf]); d > 0; d--) v *= (double)kx;
      }
      s_acc[o] = v;
    }
    __syncthreads();
    const double* Eb = A.E + B.e_off + (size_t)s_p[j] * B.nterm;
    for (int e = tid; e < NI; e += NT) {
      const int a = e / nf, f = e - a * nf;
      if (!((mask >> f) & 1)) continue;
      double s = 0.0;
      for (int x = SB.fs[a]; x < SB.fs[a + 1]; x++) s = fma(Eb[x], s_acc[sh_pack_idx(SB.term[x]) * nf + f], s);
      s_out[e] += s;
    }
    __syncthreads();
    for (int o = tid; o < NO; o += NT) s_acc[o] = 0.0;
  };

  for (int tier = 0; tier < 2; tier++) {
    const int* scan = s_scan[tier];
    const int n = scan[SH_MAXSLICE];
    for (int base = 0; base < n; base += NT) {
      // ---- 1. one item per thread ----
      const int item = base + tid;
      if (item < n) {
        int j = 0;
#pragma unroll
        for (int s = SH_MAXSLICE / 2; s > 0; s >>= 1)
          if (scan[j + s] <= item) j += s;
        const int p = s_p[j];
        const int q = item - scan[j] + (tier ? s_c64[j] : 0);
        s_q[tid] = q;
        if (tier == 0) {
          const ShPrim a = bra[p], b = ket[q];
          double pre = a.w * b.w;
          if (diag && q < p) pre = pre + pre;
          const double rs = rsqrt(a.p + b.p);
          pre *= rs;
          const double alpha = a.p * b.p * (rs * rs);
          const double m2a = -2.0 * alpha;
          double bs[L + 1];
          double* row = s_R + tid * ROW;
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
            boys_shell<L>(alpha * fma(X, X, fma(Y, Y, Z * Z)), F, s_boys, s_e2);
            double pw = pre;
#pragma unroll
            for (int m = 0; m <= L; m++) {
              bs[m] = pw * F[m];
              if (m < L) pw *= m2a;
            }
            store_row<L, double>(X, Y, Z, bs, row);
          }
        } else {
          // FP32: degree n carries a factor kx^-n (kx ~ sqrt(2p) of the bra primitive), which
          // keeps (2 alpha)^L of tight primitives inside the FP32 range
          const ShPrimF a = A.primf[B.prim_off + p], b = A.primf[K.prim_off + q];
          const float kx = H == 1 ? 1.f : a.kx;
          const float ik = 1.f / kx;
          float pre = a.w * b.w;
          const float rs = rsqrtf(a.p + b.p);
          pre *= rs;
          const float alpha = (a.p * rs) * (b.p * rs);
          const float m2a = -2.f * (alpha * ik * ik);
          float bs[L + 1];
          float* row = reinterpret_cast<float*>(s_R) + tid * ROW;
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
            boys_shell<L>(alpha * fmaf(X, X, fmaf(Y, Y, Z * Z)), F, s_boys32);
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
      // ---- 2. segments of the batch: runs of one bra primitive (an s-type bra needs none) ----
      const int top = min(base + NT, n);
      int j = 0;
#pragma unroll
      for (int s = SH_MAXSLICE / 2; s > 0; s >>= 1)
        if (scan[j + s] <= base) j += s;
      int lo = base;
      while (lo < top) {
        while (scan[j + 1] <= lo) j++;
        const int hi = H == 1 ? top : min(top, scan[j + 1]);
        const float kx = (tier && H > 1) ? A.primf[B.prim_off + s_p[j]].kx : 1.f;
        const int i0 = lo - base, i1 = hi - base;
        for (int o = my_o; o < NO && my_g < G; o += NT) {
          const int t = o / nf, f = o - t * nf;
          if ((mask >> f) & 1) {
            const uint32_t ht = sh_hermite[t];
            double acc = 0.0;
            for (int x = SK.fs[f]; x < SK.fs[f + 1]; x++) {
              const uint32_t tau = SK.term[x];
              const uint32_t tt = ht + tau;
              if (onec && (tt & 0x010101u)) continue;  // odd degrees vanish on one centre
              const int col = sh_pack_idx(tt);
              const int dt = sh_degree(tau);
              if (tier == 0) {
                const double* Ek = A.E + K.e_off + x;
                const double* Rc = s_R + col;
                double s = 0.0;
#pragma unroll 4
                for (int i = i0 + my_g; i < i1; i += G) s = fma(Rc[i * ROW], Ek[(size_t)s_q[i] * K.nterm], s);
                acc += (dt & 1) ? -s : s;
              } else {
                const float* Ek = A.Ef + K.e_off + x;
                const float* Rc = reinterpret_cast<const float*>(s_R) + col;
                float s = 0.f;
#pragma unroll 4
                for (int i = i0 + my_g; i < i1; i += G) s = fmaf(Rc[i * ROW], Ek[(size_t)s_q[i] * K.nterm], s);
                double v = (double)s;
                for (int d = 0; d < dt; d++) v *= (double)kx;
                acc += (dt & 1) ? -v : v;
              }
            }
            s_acc[o + my_g * NO] += acc;
          }
          if (NO < NT) break;
        }
        if (H > 1 && hi == scan[j + 1]) flush(j, kx);
        lo = hi;
      }
      __syncthreads();
    }
  }
  if (H == 1 && nb > 0) {
    if (tid == 0) s_p[0] = 0;
    flush(0, 1.f);
  }
  __syncthreads();
  if (diag) {
    for (int a = tid; a < nf; a += NT) A.partial[W.part + (int64_t)a * W.split + slice] = SH_PI_5_2 * s_out[a * nf + a];
  } else {
    for (int e = tid; e < NI; e += NT) A.partial[W.part + (int64_t)e * W.split + slice] = SH_PI_5_2 * s_out[e];
  }
}

template <int L>
cudaError_t launch_shell_L(int ncta, int max_no, int max_ni, cudaStream_t st, const ShArgs& A) {
  const size_t smem = ShSmem<L>::bytes(max_no, max_ni);
  if (smem > SH_SMEM_MAX) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(shell_eri_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, SH_SMEM_MAX);
  if (e != cudaSuccess) return e;
  shell_eri_kernel<L><<<ncta, ShSmem<L>::NT, smem, st>>>(A, max_no, max_ni);
  return cudaGetLastError();
}

}  // namespace ss
