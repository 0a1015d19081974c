// shell_tables.cu -- shells and shell pairs of the basis, their primitive tables, and the analytic
// ERIs of shell quartets (shell_eri.cuh).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <unordered_map>
#include <vector>

#include "boys_grid.cuh"
#include "shell_basis.h"
#include "shell_host.h"
#include "ss_context.cuh"

namespace ss {

// A kept primitive quartet whose Schwarz bound is below this part of the shell quartet's (and above
// the FP32 tier) is evaluated in two floats, the larger ones in FP64.  Measured error against plain
// 64-bit values, largest over the integrals of a system relative to their Schwarz bounds (water 7
// functions; O; O-H; H2O of 19 functions): all FP64 1.4e-15, 4.3e-15, 4.5e-15, 2.8e-15 with the
// per-function kernels; here 1e-5: 1.2e-15, 2.4e-15, 1.9e-15, 2.8e-15; 1e-4: 1.9e-15, 2.2e-15,
// 9.4e-15, 2.8e-15; 1e-3: 1.4e-14, 9.6e-15, 4.0e-14, 9.9e-15; all two-float: 2.5e-14 to 1.5e-13.
// Against 80-bit sums (water 7 functions at 20, 13, 9 Gaussians; H2; O; N; O-H), per-function kernels ->
// here: largest error 1.3e-15 -> 9.4e-16, 1.2e-15 -> 4.1e-16, 9.9e-16 -> 4.2e-16, 1.5e-15 -> 5.6e-16,
// 9.6e-16 -> 6.8e-16, 4.3e-15 -> 1.9e-15, 2.8e-15 -> 6.9e-16 of the Schwarz bound.
// About a tenth of the FP64 work is left above 1e-5.
constexpr double SH_DF_EPS = 1e-5;

#define TRY(x)           \
  do {                   \
    int rc_ = (x);       \
    if (rc_) return rc_; \
  } while (0)

// ---- device tables ---------------------------------------------------------------------------

struct ShFill {
  ShPrim* prim;
  double* E;
  int* cnt;
};

// Primitive records of one shell pair per CTA, in (m1, m2) order, the primitives with K_AB below
// the reference's cuts dropped (src/gaussian_product.F90:25-28,
// src/give_explicit_poly_and_gaussian.F90:46-49), and the Hermite coefficients of every component.
// fold: both shells have the same fit on one centre, so (m1, m2) and (m2, m1) are the same
// distribution: m1 <= m2 only, the coefficient doubled for m1 < m2 (exact).
__global__ void __launch_bounds__(256) shell_fill(BasisDev B, const ShPair* __restrict__ pairs,
                                                  const ShStruct* __restrict__ st, ShFill out) {
  const ShPair P = pairs[blockIdx.x];
  const ShStruct& S = st[P.st];
  __shared__ int s_wcnt[8], s_total;
  if (threadIdx.x == 0) s_total = 0;
  const int na = B.n_gauss[P.fa], nb = B.n_gauss[P.fb];
  const int64_t ta = B.i_type[P.fa] == 2 ? 1 : 0, tb = B.i_type[P.fb] == 2 ? 1 : 0;
  const double* A = B.center + 3 * P.fa;
  const double* C = B.center + 3 * P.fb;
  const double x0 = A[0] - C[0], x1 = A[1] - C[1], x2 = A[2] - C[2];
  const double r2 = x0 * x0 + x1 * x1 + x2 * x2;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = na * nb;
  for (int t0 = 0; t0 < n; t0 += 256) {
    const int t = t0 + threadIdx.x;
    const int m1 = t / nb, m2 = t - m1 * nb;
    bool keep = t < n && !(P.fold && m2 < m1);
    double a = 0, b = 0, K = 0;
    if (keep) {
      a = B.g_gauss[m1 + (int64_t)B.ld * P.fa];
      b = B.g_gauss[m2 + (int64_t)B.ld * P.fb];
      const double kk = (a * b) * (1.0 / (a + b)) * r2;
      K = kk > 40.0 ? 0.0 : exp(-kk);
      keep = !(kk > 40.0) && !(K < 1.e-15);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    __syncthreads();
    if (lane == 0) s_wcnt[wid] = __popc(bal);
    __syncthreads();
    int pos = s_total + __popc(bal & ((1u << lane) - 1));
    for (int w = 0; w < wid; w++) pos += s_wcnt[w];
    if (keep) {
      ShPrim r;
      r.p = a + b;
      const double p_inv = 1.0 / r.p;
      for (int ax = 0; ax < 3; ax++) r.P[ax] = P.onec ? A[ax] : (a * A[ax] + b * C[ax]) * p_inv;
      double coef = B.c_gauss[m1 + (int64_t)B.ld * (P.fa + (int64_t)B.n * ta)] *
                    B.c_gauss[m2 + (int64_t)B.ld * (P.fb + (int64_t)B.n * tb)];
      if (P.fold && m1 != m2) coef = 2.0 * coef;
      r.w = (K * coef) * p_inv;
      r.S = 0.0;
      out.prim[P.prim_off + pos] = r;
      // E^{ij}_t of the three axes (McMurchie and Davidson): E^{i+1,j}_t = E^{ij}_{t-1} / 2p +
      // PA E^{ij}_t + (t+1) E^{ij}_{t+1}, and the same in j with PB
      const double h = 0.5 * p_inv;
      double e[3][3][3][5];
      for (int ax = 0; ax < 3; ax++) {
        const double pa = P.onec ? 0.0 : r.P[ax] - A[ax], pb = P.onec ? 0.0 : r.P[ax] - C[ax];
        for (int i = 0; i < 3; i++)
          for (int j = 0; j < 3; j++) {
            for (int u = 0; u < 5; u++) {
              double v = 0.0;
              if (i == 0 && j == 0) {
                v = u == 0 ? 1.0 : 0.0;
              } else {
                const double* s = j > 0 ? e[ax][i][j - 1] : e[ax][i - 1][0];
                const double x = j > 0 ? pb : pa;
                v = x * s[u];
                if (u > 0) v = fma(h, s[u - 1], v);
                if (u < 4) v = fma((double)(u + 1), s[u + 1], v);
              }
              e[ax][i][j][u] = v;
            }
          }
      }
      double* E = out.E + P.e_off + (size_t)pos * P.nterm;
      for (int f = 0; f < S.ncomp; f++)
        for (int x = S.fs[f]; x < S.fs[f + 1]; x++) {
          const uint32_t tm = S.term[x];
          double v = 0.0;
          for (int k = 0; k < S.ncombo[f]; k++) {
            const uint32_t c = S.combo[f][k];
            const double ex = e[0][c & 15][(c >> 12) & 15][tm & 255];
            const double ey = e[1][(c >> 4) & 15][(c >> 16) & 15][(tm >> 8) & 255];
            const double ez = e[2][(c >> 8) & 15][(c >> 20) & 15][tm >> 16];
            v += ex * ey * ez;
          }
          E[x] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < 8; w++) s_total += s_wcnt[w];
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) out.cnt[blockIdx.x] = s_total;
}

// sum of the partial sums of every element: one warp per element, lane sums and a shuffle tree
__global__ void __launch_bounds__(256) shell_reduce(int nwork, const ShWork* __restrict__ work,
                                                    const ShPair* __restrict__ pairs, int diag,
                                                    const double* __restrict__ part, double* __restrict__ elem) {
  const ShWork W = work[blockIdx.x];
  const int ni = diag ? pairs[W.bra].ncomp : pairs[W.bra].ncomp * pairs[W.ket].ncomp;
  const int n = W.split + W.lsplit, lane = threadIdx.x & 31;
  for (int e = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5); e < ni; e += gridDim.y * (blockDim.x >> 5)) {
    const double* p = part + W.part + (int64_t)e * n;
    double v = 0.0;
    for (int s = lane; s < n; s += 32) v = v + p[s];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) elem[W.elem + e] = v;
  }
}

// work entry of every CTA
__global__ void shell_expand(const ShWork* __restrict__ work, int* __restrict__ cta, int* __restrict__ lcta) {
  const ShWork W = work[blockIdx.x];
  for (int s = threadIdx.x; s < W.split; s += blockDim.x) cta[W.cta0 + s] = blockIdx.x;
  for (int s = threadIdx.x; s < W.nlane; s += blockDim.x) lcta[W.lcta0 + s] = blockIdx.x;
}

// exponent of the largest power of two whose square is at most 2 p, and a power of two, from the bits
// of the double (normal numbers; with ilogb and ldexp the sort took 0.28 ms instead of 0.21 for the
// 26-function water)
__device__ __forceinline__ int unit_exp(double p) {
  return ((int)((uint64_t)__double_as_longlong(p + p) >> 52) - 1023) >> 1;
}
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((int64_t)(1023 + e) << 52); }

// Schwarz factors of a pair's primitives and their sorted tables.  A primitive's factor is the
// largest over the components of sqrt((P_f|P_f) / (f|f)), (f|f) the contracted diagonal: then
// |(P_f|Q_g)| <= S_P S_Q sqrt((f|f)(g|g)) for every pair of components.  A component without a
// positive diagonal keeps all its primitives (factor 1e30).  Sorted by decreasing factor (ties:
// the (m1, m2) order), with a two-float copy of the records and coefficients whose w is divided by
// a power of two near the square root of the pair's largest diagonal, so that the FP32 evaluations
// of distant (small) pairs stay inside the FP32 range.
__global__ void __launch_bounds__(512) shell_sort(const ShPair* __restrict__ pairs, const ShStruct* __restrict__ st,
                                                  const int* __restrict__ cnt, const double* __restrict__ diag,
                                                  const ShPrim* __restrict__ prim, const double* __restrict__ E,
                                                  ShPrim* __restrict__ oprim, ShPrimF* __restrict__ oprimf,
                                                  double* __restrict__ oE, float2* __restrict__ oE2,
                                                  double* __restrict__ oscale) {
  __shared__ double s_key[1024];
  __shared__ int s_idx[1024];
  const ShPair P = pairs[blockIdx.x];
  const ShStruct& S = st[P.st];
  const int m = cnt[blockIdx.x];
  for (int t = threadIdx.x; t < 1024; t += blockDim.x) {
    double key = -1.0;
    if (t < m) {
      const ShPrim a = prim[P.prim_off + t];
      const double* e = E + P.e_off + (size_t)t * P.nterm;
      // (P|P): both on one centre at exponent p/2, so R_{2a 2b 2c} = (2a-1)!!(2b-1)!!(2c-1)!! (-p)^n / (2n+1)
      const double pre = 34.9868366552 * a.w * a.w * rsqrt(a.p + a.p);
      double pw[SH_MAXL / 2 + 1];
      pw[0] = 1.0;
#pragma unroll
      for (int n = 1; n <= SH_MAXL / 2; n++) pw[n] = pw[n - 1] * -a.p;
#pragma unroll
      for (int n = 1; n <= SH_MAXL / 2; n++) pw[n] *= 1.0 / (2 * n + 1);
      key = 0.0;
      for (int f = 0; f < S.ncomp; f++) {
        double v = 0.0;
        for (int x = S.fs[f]; x < S.fs[f + 1]; x++) {
          double row = 0.0;
          for (int y = S.fs[f]; y < S.fs[f + 1]; y++) {
            const uint32_t h = S.term[x] + S.term[y];
            if (h & 0x010101u) continue;
            const int hx = h & 255, hy = (h >> 8) & 255, hz = h >> 16;
            // (2a-1)!! = 1, 1, 3, 15, 105
            auto dfact = [](int e) { return e <= 2 ? 1.f : e == 4 ? 3.f : e == 6 ? 15.f : 105.f; };
            const int n = (hx + hy + hz) / 2;
            double r = pw[0];
#pragma unroll
            for (int t = 1; t <= SH_MAXL / 2; t++) r = t == n ? pw[t] : r;
            const int dy = (S.term[y] & 255) + ((S.term[y] >> 8) & 255) + (S.term[y] >> 16);
            const float c = dfact(hx) * dfact(hy) * dfact(hz);
            row = fma(r * (double)((dy & 1) ? -c : c), e[y], row);
          }
          v = fma(row, e[x], v);
        }
        const double d = diag[(size_t)blockIdx.x * SH_MAXCOMP + f];
        const double s = d > 0.0 ? sqrt(fmax(pre * v, 0.0) / d) : 1e30;
        key = fmax(key, s < 1e30 ? s : 1e30);  // also where the quotient overflowed or is not a number
      }
    }
    s_key[t] = key;
    s_idx[t] = t;
  }
  __syncthreads();
  for (int k = 2; k <= 1024; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < 1024; t += blockDim.x) {
        const int u = t ^ j;
        if (u > t) {
          const bool up = (t & k) == 0;
          const bool first = s_key[t] > s_key[u] || (s_key[t] == s_key[u] && s_idx[t] < s_idx[u]);
          if (up != first) {
            const double kk = s_key[t];
            const int ii = s_idx[t];
            s_key[t] = s_key[u]; s_idx[t] = s_idx[u];
            s_key[u] = kk; s_idx[u] = ii;
          }
        }
      }
      __syncthreads();
    }
  double dmax = 0.0;
  for (int f = 0; f < S.ncomp; f++) dmax = fmax(dmax, diag[(size_t)blockIdx.x * SH_MAXCOMP + f]);
  const int ex = dmax > 0.0 ? ilogb(dmax) / 2 : 0;
  if (threadIdx.x == 0) oscale[blockIdx.x] = ldexp(1.0, ex);
  for (int t = threadIdx.x; t < m; t += blockDim.x) {
    ShPrim a = prim[P.prim_off + s_idx[t]];
    a.S = s_key[t];
    oprim[P.prim_off + t] = a;
    auto two = [](double v, float* hi, float* lo) {
      *hi = (float)v;
      *lo = (float)(v - (double)*hi);
    };
    ShPrimF g;
    two(a.p, &g.p[0], &g.p[1]);
    two(ldexp(a.w, -ex), &g.w[0], &g.w[1]);
    for (int ax = 0; ax < 3; ax++) {
      two(a.P[ax], &g.ph[ax], &g.pl[ax]);
      g.pm[ax] = (float)((a.P[ax] - (double)g.ph[ax]) - (double)g.pl[ax]);
    }
    g.pad = 0.f;
    g.s = (float)pow2(unit_exp(a.p));
    g.is = (float)pow2(-unit_exp(a.p));
    oprimf[P.prim_off + t] = g;
  }
  for (int t = threadIdx.x; t < m * P.nterm; t += blockDim.x) {
    const int r = t / P.nterm, x = t - r * P.nterm;
    const double v = E[P.e_off + (size_t)s_idx[r] * P.nterm + x];
    oE[P.e_off + t] = v;
    const uint32_t tm = S.term[x];
    const int deg = (int)((tm & 255) + ((tm >> 8) & 255) + (tm >> 16));
    const double u = v * pow2(deg * unit_exp(prim[P.prim_off + s_idx[r]].p));
    const float hi = (float)u;
    oE2[P.e_off + t] = make_float2(hi, (float)(u - (double)hi));
  }
}

// Boys tables of every top degree (ShBoys), from the grid F_n(T_k)
__global__ void shell_boys(ShBoys* __restrict__ out) {
  const int L = blockIdx.y, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= SH_BOYS_K) return;
  double fact = 1.0;
  float* f = out[L].f[k];
  for (int j = 0; j < 9; j++) {
    if (j > 1) fact *= j;
    const double a = boys_grid_tab[k * BOYS_GRID_N + L + j] / fact;
    out[L].a[k][j] = a;
    if (j < 5) {
      f[2 * j] = (float)a;
      f[2 * j + 1] = (float)(a - (double)(float)a);
    } else {
      f[12 + j - 5] = (float)a;
    }
  }
  const double e = exp(-0.125 * k);
  f[10] = (float)e;
  f[11] = (float)(e - (double)(float)e);
  for (int j = 16; j < SH_BOYS_ROW; j++) f[j] = 0.f;
}

#define SH_DECL(L) cudaError_t launch_shell_##L(int, int, int, int, cudaStream_t, const ShArgs&);
SH_DECL(0) SH_DECL(1) SH_DECL(2) SH_DECL(3) SH_DECL(4) SH_DECL(5) SH_DECL(6) SH_DECL(7) SH_DECL(8)
#undef SH_DECL

cudaError_t launch_shell_eri(int L, int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A) {
  switch (L) {
#define SH_CASE(l) case l: return launch_shell_##l(ncta, max_no, max_ni, max_col, st, A);
    SH_CASE(0) SH_CASE(1) SH_CASE(2) SH_CASE(3) SH_CASE(4) SH_CASE(5) SH_CASE(6) SH_CASE(7) SH_CASE(8)
#undef SH_CASE
  }
  return cudaErrorInvalidValue;
}

#define SH_LANE_KETS(X) \
  X(ss, SH_S, SH_S) X(ps, SH_P, SH_S) X(pp, SH_P, SH_P) X(rs, SH_R, SH_S) X(rp, SH_R, SH_P) X(rr, SH_R, SH_R) \
  X(ds, SH_D, SH_S) X(dr, SH_D, SH_R)
#define SH_DECL(n, a, b)                                                     \
  cudaError_t launch_lane_##n(int, int, cudaStream_t, const ShArgs&);        \
  cudaError_t launch_lane_##n##1(int, int, cudaStream_t, const ShArgs&);     \
  cudaError_t launch_lane_##n##4(int, int, cudaStream_t, const ShArgs&);
SH_LANE_KETS(SH_DECL)
#undef SH_DECL
cudaError_t launch_lane_pps(int, int, cudaStream_t, const ShArgs&);
cudaError_t launch_lane_pps4(int, int, cudaStream_t, const ShArgs&);
// an s pair has one term on one and on two centres
cudaError_t launch_lane_ss1(int db, int ncta, cudaStream_t st, const ShArgs& A) { return launch_lane_ss(db, ncta, st, A); }

cudaError_t launch_shell_lane(int instance, int ncta, cudaStream_t st, const ShArgs& A) {
  const bool all = instance >= SH_LANE_ONEC;
  const int db = instance & 7, ket = (instance & (SH_LANE_ONEC - 1)) >> 3;
#define SH_CASE(n, a, b)                                                          \
  if (ket / 2 == a * (a + 1) / 2 + b)                                             \
    return all ? launch_lane_##n##4(db, ncta, st, A) : (ket & 1) ? launch_lane_##n##1(db, ncta, st, A) \
                                                                 : launch_lane_##n(db, ncta, st, A);
  SH_LANE_KETS(SH_CASE)
#undef SH_CASE
  if (ket / 2 == SH_NBASE) return all ? launch_lane_pps4(db, ncta, st, A) : launch_lane_pps(db, ncta, st, A);
  return cudaErrorInvalidValue;
}

// ---- host ------------------------------------------------------------------------------------

// multiply-adds of the Hermite integrals of total degree L
static const double SH_REC[SH_MAXL + 1] = {2, 8, 24, 60, 120, 200, 330, 520, 790};

// pair type (without the one-centre bit) of the lane kernels' rule
static int lane_chunk(const ShPair& b, const ShPair& k) {
  const int base = k.st / 2;
  if (base == SH_NBASE + 1) return 0;  // D with itself
  const int ix = base == SH_NBASE ? SH_P * (SH_P + 1) / 2 + SH_P : base;
  for (int ta = 0; ta < 4; ta++)
    for (int tb = 0; tb <= ta; tb++)
      if (ta * (ta + 1) / 2 + tb == ix) return sh_lane_chunk(b.d, ta, tb);
  return 0;
}

// FP32-pipe instructions of one primitive quartet in two floats with this bra and ket: the Hermite
// integrals (once per chunk of the ket's components in the lane kernels), a two-float
// multiply-add per bra Hermite function and ket term, and the shared kernel's own overhead
// (loads and indices per term, barriers and segments).  The cheaper orientation is taken.
static double side_cost(const ShPair& b, const ShPair& k) {
  const int L = b.d + k.d;
  const double herm = 290.0 + 36.0 * L + 8.0 * SH_REC[L], terms = (double)sh_nherm(b.d) * k.nterm;
  const int c = lane_chunk(b, k);
  return c ? herm * ((k.ncomp + c - 1) / c) + 12.2 * terms : herm + 18.0 * terms + 1500.0;
}

// bra slices of a shell quartet in the shared kernel: two to eight bra primitives per CTA (about 1e6
// multiply-adds at a hundred kept kets each), 16 where it only has the FP64 tier; never from what
// else is in the list, so that the order of summation is the quartet's own.  On a small system the
// longest CTA is the stage, on a large one a CTA's start-up counts: at most 4, 8, 16 primitives took
// 2.37, 2.43, 2.50 ms for the oxygen atom and 45.0, 44.3, 44.0 ms for the 26-function water.
static int slices(const ShPair& b, const ShPair& k, bool lane) {
  const int L = b.d + k.d;
  const double cost = 30.0 + 4.0 * L + SH_REC[L] + (double)sh_nherm(b.d) * k.nterm;
  const int per = lane ? SH_MAXSLICE : (int)std::min(8.0, std::max(2.0, 1e4 / cost));
  return std::max(1, (b.cap + per - 1) / per);
}

// Launch the work entries (grouped by total degree), in chunks whose partial sums fit the buffer,
// and reduce each chunk's partial sums to elements.  All chunks' entries go up in one copy before the
// first launch, so that the host waits for no chunk's kernels.
static int run_work(ss_ctx* c, ShellPlan& Lw, const ShPrim* prim, const ShPrimF* primf, const double* E, const float2* E2,
                    bool diag, double eps, double eps32, double* elem) {
  const ShellBasis& T = c->shells;
  // partial sums in flight: enough for a whole mid-size system, and bounded
  size_t cap = (size_t)64 << 20;
  if (c->budget) cap = std::min(cap, std::max<size_t>((c->budget - std::min(c->budget, c->used)) / 4, 1 << 20));
  const int64_t cap_d = (int64_t)(cap / sizeof(double));
  struct Seg { int L, cta0, ncta, no, ni, col; };
  struct LaneSeg { int instance, cta0, ncta; };
  struct Chunk {
    size_t first, n = 0;
    int64_t part = 0;
    int ncta = 0, nlane = 0;
    std::vector<Seg> segs;
    std::vector<LaneSeg> lanes;
    explicit Chunk(size_t f) : first(f) {}
  };
  std::vector<ShWork> work;
  std::vector<Chunk> chunks;
  // heaviest degrees first: their CTAs are the longest
  for (int L = SH_MAXL; L >= 0; L--) {
    std::vector<ShWork>& v = Lw.work[L];
    auto cost = [&](const ShWork& w) { return side_cost(T.pair[w.bra], T.pair[w.ket]); };
    std::stable_sort(v.begin(), v.end(), [&](const ShWork& a, const ShWork& b) { return cost(a) > cost(b); });
    bool open = false;
    for (ShWork w : v) {
      const ShPair &b = T.pair[w.bra], &k = T.pair[w.ket];
      const int ni = b.ncomp * k.ncomp;
      const int64_t need = (int64_t)(w.split + w.lsplit) * (diag ? b.ncomp : ni);
      if (chunks.empty() || (chunks.back().n && (chunks.back().part + need > cap_d ||
                                                 chunks.back().ncta + chunks.back().nlane > (1 << 28)))) {
        chunks.emplace_back(work.size());
        open = false;
      }
      Chunk& C = chunks.back();
      if (!open) {
        C.segs.push_back(Seg{L, C.ncta, 0, 0, 0, 0});
        open = true;
      }
      Seg& g = C.segs.back();
      w.cta0 = C.ncta;
      w.part = C.part;
      work.push_back(w);
      g.ncta += w.split;
      g.no = std::max(g.no, sh_nherm(b.d) * k.ncomp);
      g.ni = std::max(g.ni, ni);
      g.col = std::max(g.col, sh_col_size(b.d, k.nterm));
      C.n++;
      C.ncta += w.split;
      C.nlane += w.nlane;
      C.part += need;
    }
  }
  if (chunks.empty()) return SS_OK;
  int64_t part = 0, ctas = 0;
  for (Chunk& C : chunks) {
    // the lane kernels' CTAs, an instance's together
    std::vector<size_t> order;
    for (size_t t = C.first; t < C.first + C.n; t++)
      if (work[t].lane >= 0) order.push_back(t);
    std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) { return work[x].lane > work[y].lane; });
    int nlane = 0;
    for (size_t t : order) {
      if (C.lanes.empty() || C.lanes.back().instance != work[t].lane) C.lanes.push_back(LaneSeg{work[t].lane, nlane, 0});
      work[t].lcta0 = nlane;
      C.lanes.back().ncta += work[t].nlane;
      nlane += work[t].nlane;
    }
    part = std::max(part, C.part);
    ctas = std::max(ctas, (int64_t)C.ncta + C.nlane);
  }
  void *dc, *dp;
  TRY(pool_get(c, "shell_part", sizeof(double) * (size_t)part, &dp));
  TRY(pool_get(c, "shell_cta", sizeof(int) * (size_t)ctas, &dc));
  TRY(h2d_async(c, c->pool["shell_work"], work.data(), sizeof(ShWork) * work.size()));
  const ShWork* dwork = (const ShWork*)c->pool["shell_work"].ptr;
  ShArgs A{};
  A.pair = (const ShPair*)c->pool["shell_pair"].ptr;
  A.cnt = (const int*)c->pool["shell_cnt"].ptr;
  A.st = (const ShStruct*)c->pool["shell_struct"].ptr;
  A.prim = prim;
  A.primf = primf;
  A.E = E;
  A.E2 = E2;
  A.scale = (const double*)c->pool["shell_scale"].ptr;
  A.boys = (const ShBoys*)c->pool["shell_boys"].ptr;
  A.col = (const uint8_t*)c->pool["shell_col"].ptr;
  A.partial = (double*)dp;
  A.eps = eps;
  A.eps32 = eps32;
  A.eps_df = SH_DF_EPS;
  A.diag = diag;
  A.cta = (const int*)dc;
  for (const Chunk& C : chunks) {
    A.work = dwork + C.first;
    int* lcta = (int*)dc + C.ncta;
    A.lcta = lcta;
    shell_expand<<<(unsigned)C.n, 32, 0, c->stream>>>(A.work, (int*)dc, lcta);
    SS_CUDA_TRY(cudaGetLastError());
    c->launches++;
    TRY(fork_eri_streams(c));
    int rc = SS_OK;
    size_t launch = 0;
    for (size_t s = 0; s < C.lanes.size() && !rc; s++) {
      A.cta0 = C.lanes[s].cta0;
      const cudaError_t e = launch_shell_lane(C.lanes[s].instance, C.lanes[s].ncta, c->eri_stream[launch++ % ss_ctx::ERI_STREAMS], A);
      if (e != cudaSuccess) {
        ss_set_cuda_error(e, "shell_lane_kernel launch", __FILE__, __LINE__);
        rc = SS_ERR_CUDA;
      }
      c->launches++;
    }
    for (size_t s = 0; s < C.segs.size() && !rc; s++) {
      const Seg& g = C.segs[s];
      A.cta0 = g.cta0;
      const cudaError_t e = launch_shell_eri(g.L, g.ncta, g.no, g.ni, g.col, c->eri_stream[launch++ % ss_ctx::ERI_STREAMS], A);
      if (e != cudaSuccess) {
        ss_set_cuda_error(e, "shell_eri_kernel launch", __FILE__, __LINE__);
        rc = SS_ERR_CUDA;
      }
      c->launches++;
    }
    const int jrc = join_eri_streams(c);
    if (rc || jrc) return rc ? rc : jrc;
    shell_reduce<<<dim3((unsigned)C.n, 4), 256, 0, c->stream>>>((int)C.n, A.work, A.pair, diag, (const double*)dp, elem);
    SS_CUDA_TRY(cudaGetLastError());
    c->launches++;
  }
  return SS_OK;
}

// Primitive tables of the shell pairs and the Schwarz diagonal (ik|ik) of every function pair in
// shells, into the host matrix pre (n x n); other pairs' entries are left as they are.
int shell_precond(ss_ctx* c, std::vector<double>& pre) {
  const ShellBasis& T = c->shells;
  const int np = (int)T.pair.size();
  if (!np) return SS_OK;
  void* p;
  if (!c->have_shell_consts) {  // once per context; a call that failed half-way left the flag unset
    TRY(pool_get(c, "shell_struct", sizeof(ShStruct) * SH_NSTRUCT, &p));
    TRY(h2d_copy(c, p, structs().s.data(), sizeof(ShStruct) * SH_NSTRUCT));
    TRY(pool_get(c, "shell_col", structs().col.size(), &p));
    TRY(h2d_copy(c, p, structs().col.data(), structs().col.size()));
    TRY(pool_get(c, "shell_boys", sizeof(ShBoys) * (SH_MAXL + 1), &p));
    shell_boys<<<dim3((SH_BOYS_K + 63) / 64, SH_MAXL + 1), 64, 0, c->stream>>>((ShBoys*)p);
    SS_CUDA_TRY(cudaGetLastError());
    c->launches++;
    c->have_shell_consts = true;
  }
  const ShStruct* st = (const ShStruct*)c->pool["shell_struct"].ptr;
  TRY(h2d_async(c, c->pool["shell_pair"], T.pair.data(), sizeof(ShPair) * np));
  const ShPair* dpair = (const ShPair*)c->pool["shell_pair"].ptr;
  ShFill F;
  int* cnt;
  double *E2, *diag;
  ShPrim* prim2;
  ShPrimF* primf;
  float2* E2f;
  double* scale;
  TRY(pool_get(c, "shell_prim0", sizeof(ShPrim) * T.nprim, &p)); F.prim = (ShPrim*)p;
  TRY(pool_get(c, "shell_E0", sizeof(double) * T.nE, &p)); F.E = (double*)p;
  TRY(pool_get(c, "shell_cnt", sizeof(int) * np, &p)); F.cnt = cnt = (int*)p;
  TRY(pool_get(c, "shell_prim", sizeof(ShPrim) * T.nprim, &p)); prim2 = (ShPrim*)p;
  TRY(pool_get(c, "shell_primf", sizeof(ShPrimF) * T.nprim, &p)); primf = (ShPrimF*)p;
  TRY(pool_get(c, "shell_E", sizeof(double) * T.nE, &p)); E2 = (double*)p;
  TRY(pool_get(c, "shell_E2", sizeof(float2) * T.nE, &p)); E2f = (float2*)p;
  TRY(pool_get(c, "shell_scale", sizeof(double) * np, &p)); scale = (double*)p;
  TRY(pool_get(c, "shell_diag", sizeof(double) * np * SH_MAXCOMP, &p)); diag = (double*)p;
  SS_CUDA_TRY(cudaMemsetAsync(diag, 0, sizeof(double) * np * SH_MAXCOMP, c->stream));
  shell_fill<<<np, 256, 0, c->stream>>>(c->basis, dpair, st, F);
  SS_CUDA_TRY(cudaGetLastError());
  c->launches++;
  ShellPlan Lw;
  for (int x = 0; x < np; x++) {
    const ShPair& P = T.pair[x];
    if (P.cap == 0) continue;  // (ik|ik) = 0
    ShWork w{};
    w.bra = w.ket = x;
    w.split = std::max(1, (P.cap + 1) / 2);  // two bra primitives: few quartets, in FP64
    w.lane = -1;
    w.elem = (int64_t)x * SH_MAXCOMP;
    w.mask = ~0ull;
    Lw.work[2 * P.d].push_back(w);
  }
  TRY(run_work(c, Lw, F.prim, nullptr, F.E, nullptr, true, 0.0, 0.0, diag));
  shell_sort<<<np, 512, 0, c->stream>>>(dpair, st, cnt, diag, F.prim, F.E, prim2, primf, E2, E2f, scale);
  SS_CUDA_TRY(cudaGetLastError());
  c->launches++;
  std::vector<double> h((size_t)np * SH_MAXCOMP);
  SS_CUDA_TRY(cudaMemcpyAsync(h.data(), diag, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, c->stream));
  SS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const int n = c->n;
  for (int i = 0, f0 = 0; i < n; i++) {
    if (!c->h_sys.empty() && c->h_sys[i] != c->h_sys[f0]) f0 = i;  // first function of the system
    for (int k = f0; k <= i; k++) {
      int pr, f;
      if (!T.component(i, k, &pr, &f)) continue;
      pre[i + (size_t)n * k] = pre[k + (size_t)n * i] = h[(size_t)pr * SH_MAXCOMP + f];
    }
  }
  return SS_OK;
}

// Shell quartets of the selected function quartets.  Quartets with a function in no shell go to
// `rest`; of the others, slot[q] receives the place of the result (one element, offset from
// `first`), and *nelem the number of elements.  tiers: the FP32 tiers are on.
int shell_plan(ss_ctx* c, bool tiers, const std::vector<int64_t>& sel, std::vector<int64_t>& slot, std::vector<int64_t>& rest,
               ShellPlan& plan, int64_t* nelem) {
  const ShellBasis& T = c->shells;
  const int n = c->n;
  auto sys = [&](int f) { return c->h_sys.empty() ? 0 : c->h_sys[f]; };
  // shell pair and component of every two functions of a system
  std::vector<int> f0(n);
  std::vector<int64_t> row(n);
  std::vector<int32_t> fpair;
  std::vector<int16_t> fcomp;
  for (int i = 0; i < n; i++) {
    f0[i] = i > 0 && sys(i) == sys(i - 1) ? f0[i - 1] : i;
    row[i] = (int64_t)fpair.size() - f0[i];
    for (int k = f0[i]; k <= i; k++) {
      int pr = -1, f = 0;
      T.component(i, k, &pr, &f);
      fpair.push_back(pr);
      fcomp.push_back((int16_t)f);
    }
  }
  // entry of Q of every two pairs of a system, and of those across systems that the list has
  const int nsys = (int)T.first.size() - 1;
  std::vector<int64_t> block(nsys + 1, 0);
  std::vector<int> psys(T.pair.size());
  for (int s = 0; s < nsys; s++) {
    const int64_t np = T.pfirst[s + 1] - T.pfirst[s];
    block[s + 1] = block[s] + np * (np + 1) / 2;
    std::fill(psys.begin() + T.pfirst[s], psys.begin() + T.pfirst[s + 1], s);
  }
  const bool dense = block[nsys] <= (int64_t)64 << 20;
  std::vector<int32_t> where(dense ? block[nsys] : 0, -1);
  std::unordered_map<int64_t, int32_t> sparse;
  struct Quartet { int bra, ket; uint64_t mask; int64_t elem; };
  std::vector<Quartet> Q;
  int64_t elem = 0;
  for (int64_t t : sel) {
    const int i = c->h_is[t] - 1, k = c->h_ks[t] - 1, j = c->h_js[t] - 1, l = c->h_ls[t] - 1;
    if (k < f0[i] || l < f0[j]) continue;  // a product of functions of two systems is none: 0
    const int64_t a = row[i] + k, b = row[j] + l;
    const int pa = fpair[a], pb = fpair[b];
    if (pa < 0 || pb < 0) {
      rest.push_back(t);
      continue;
    }
    const int64_t hi = std::max(pa, pb), lo = std::min(pa, pb);
    int32_t* w;
    if (dense && psys[hi] == psys[lo]) {
      const int64_t h = hi - T.pfirst[psys[hi]];
      w = &where[block[psys[hi]] + h * (h + 1) / 2 + (lo - T.pfirst[psys[hi]])];
    } else {
      w = &sparse.emplace(hi * (hi + 1) / 2 + lo, -1).first->second;
    }
    if (*w < 0) {
      *w = (int32_t)Q.size();
      const ShPair &x = T.pair[hi], &y = T.pair[lo];
      const bool fwd = side_cost(x, y) <= side_cost(y, x);  // the cheaper side as the bra
      Q.push_back(Quartet{(int)(fwd ? hi : lo), (int)(fwd ? lo : hi), 0, elem});
      elem += (int64_t)x.ncomp * y.ncomp;
    }
    Quartet& s = Q[*w];
    const int nf = T.pair[s.ket].ncomp;
    const int fb = pa == s.bra ? fcomp[a] : fcomp[b], fk = pa == s.bra ? fcomp[b] : fcomp[a];
    s.mask |= 1ull << fk;
    slot[t] = (s.elem + (int64_t)fb * nf + fk) << SLOT_SPLIT_BITS | 1;
  }
  for (const Quartet& s : Q) {
    ShWork w{};
    w.bra = s.bra;
    w.ket = s.ket;
    const ShPair &b = T.pair[s.bra], &k = T.pair[s.ket];
    const int chunk = tiers && b.cap && k.cap ? lane_chunk(b, k) : 0;
    w.lane = -1;
    if (chunk) {
      bool all = b.onec && k.onec;
      for (int ax = 0; ax < 3; ax++) all = all && c->h_center[3 * b.fa + ax] == c->h_center[3 * k.fa + ax];
      w.lane = 8 * k.st + b.d + (all ? SH_LANE_ONEC : 0);
      const int kets = sh_lane_kets(b.d + k.d);
      w.nkc = (k.cap + kets - 1) / kets;
      w.lsplit = w.nkc * ((b.cap + SH_LANE_BRA - 1) / SH_LANE_BRA);
      w.nlane = w.lsplit * ((k.ncomp + chunk - 1) / chunk);
    }
    w.split = slices(b, k, chunk > 0);
    w.elem = s.elem;
    w.mask = s.mask;
    plan.work[T.pair[s.bra].d + T.pair[s.ket].d].push_back(w);
  }
  *nelem = elem;
  return SS_OK;
}

int shell_run(ss_ctx* c, ShellPlan& plan, double eps, double eps32, double* elem) {
  return run_work(c, plan, (const ShPrim*)c->pool["shell_prim"].ptr, (const ShPrimF*)c->pool["shell_primf"].ptr,
                  (const double*)c->pool["shell_E"].ptr, (const float2*)c->pool["shell_E2"].ptr, false, eps, eps32, elem);
}

}  // namespace ss
