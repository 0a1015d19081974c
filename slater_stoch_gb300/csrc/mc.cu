// mc.cu -- ZV-MC correction kernels: walker sampler, faithful per-pair ZV map and densities,
// FP64 / REF32 accumulation, block statistics (replaces src/two_e_slater.F90:386-496).
#include <math.h>

#include "philox.cuh"
#include "ss_common.cuh"
#include "mc.cuh"

namespace ss {

// ---------------------------------------------------------------------------------------
// walkers
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void walker_normals(uint64_t seed, int64_t s, double (&n)[6]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    uint32_t c[4] = {(uint32_t)s, (uint32_t)((uint64_t)s >> 32), (uint32_t)j, STREAM_WALKER};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    n[2 * j] = normcdfinv(u01_open(c[0], c[1]));
    n[2 * j + 1] = normcdfinv(u01_open(c[2], c[3]));
  }
}

// r1, r2: [3*S] walker-major.  Standard normals as draw_configuration returns.
__global__ void draw_walkers_kernel(uint64_t seed, int64_t first, int64_t S, double* __restrict__ r1,
                                    double* __restrict__ r2) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= S) return;
  double n[6];
  walker_normals(seed, first + s, n);
  r1[3 * s] = n[0]; r1[3 * s + 1] = n[1]; r1[3 * s + 2] = n[2];
  r2[3 * s] = n[3]; r2[3 * s + 1] = n[4]; r2[3 * s + 2] = n[5];
}

// per walker: |r1|, |r2|, pi_0 (src/compute_jacobian_and_pi0.F90:12-18)
__global__ void walker_aux_kernel(int64_t S, const double* __restrict__ r1, const double* __restrict__ r2,
                                  double* __restrict__ r1m, double* __restrict__ r2m, double* __restrict__ pi0) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= S) return;
  const double fpi0 = 1.0 / ((2.0 * M_PI) * (2.0 * M_PI) * (2.0 * M_PI));
  double a0 = r1[3 * s], a1 = r1[3 * s + 1], a2 = r1[3 * s + 2];
  double b0 = r2[3 * s], b1 = r2[3 * s + 1], b2 = r2[3 * s + 2];
  double m1 = a0 * a0 + a1 * a1 + a2 * a2;
  double m2 = b0 * b0 + b1 * b1 + b2 * b2;
  r1m[s] = sqrt(m1);
  r2m[s] = sqrt(m2);
  pi0[s] = exp(-0.5 * (m1 + m2)) * fpi0;
}

// ---------------------------------------------------------------------------------------
// pair densities (src/compute_densities.F90, src/u_orb.F90, src/u_gauss.F90)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ double u_orb(int nsto, double g, double r) {
  switch (nsto) {  // c_contract = 1 (src/read_basis.F90:35)
    case 0: return exp(-g * r);
    case 1: return r * exp(-g * r);
    case 2: return (r * r) * exp(-g * r);
    case 3: return (r * r) * r * exp(-g * r);
    case 4: { double r2 = r * r; return r2 * r2 * exp(-g * r); }
    default: return pow(r, (double)nsto) * exp(-g * r);
  }
}

__device__ __forceinline__ double u_gauss(const BasisDev& B, int i, double r) {
  const double r2 = r * r;
  double u = 0.0;
  const int ng = B.n_gauss[i];
  const double* c1 = B.c_gauss + (int64_t)B.ld * i;
  const double* c2 = B.c_gauss + (int64_t)B.ld * (i + (int64_t)B.n);
  const double* g = B.g_gauss + (int64_t)B.ld * i;
  for (int m = 0; m < ng; m++) u = u + (c1[m] + c2[m] * r2) * exp(-g[m] * r2);
  return u;
}

// distance from the function's centre
__device__ __forceinline__ double centre_offset(const BasisDev& B, int f, const double (&u)[3], double (&d)[3]) {
  const double* c = B.center + 3 * f;
#pragma unroll
  for (int l = 0; l < 3; l++) d[l] = u[l] - c[l];
  return sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
}

__device__ __forceinline__ double poly(const BasisDev& B, int f, const double (&d)[3]) {
  double v = 1.0;
#pragma unroll
  for (int l = 0; l < 3; l++)
    for (int t = 0; t < B.npower[3 * f + l]; t++) v = v * d[l];
  return v;
}

// One thread per (walker, pair group, electron): ZV map (src/two_e_slater.F90:406-411), densities,
// Jacobians (src/compute_jacobian_and_pi0.F90:22-30).  The pairs of a group, all components of two
// shells, share the map and the radial parts (20 exponentials each in FP64, the cost of this
// kernel, whose FP64 pipe is 85 % busy); with one thread per pair the 26-function water evaluated
// them 3.9 times as often (16,000 walkers: 5.0 ms).
// FP64 mode folds the Jacobians and 1/pi_0 into the density columns; REF32 mode keeps them apart
// for the single-precision weight of src/two_e_slater.F90:442.
template <int MODE>
__global__ void zv_pair_kernel(BasisDev B, ZvPairs P, int64_t S, const double* __restrict__ r1,
                               const double* __restrict__ r2, const double* __restrict__ r1m,
                               const double* __restrict__ r2m, const double* __restrict__ pi0,
                               ZvChunk Z) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int g = blockIdx.y;
  if (s >= S) return;
  const int i = P.i[g], k = P.k[g];
  const bool same = P.same[g] != 0;
  const double fzv = P.fzv[g], fjac = P.fjac[g];
  const int64_t og = (int64_t)g * Z.ld + s;
  const int e = blockIdx.z;
  const double* r = e == 0 ? r1 : r2;
  const double am = e == 0 ? r1m[s] : r2m[s];
  double u[3];
#pragma unroll
  for (int l = 0; l < 3; l++) u[l] = fzv * r[3 * s + l] * am + P.G[3 * g + l];
  (e == 0 ? Z.u1x : Z.u2x)[og] = u[0];
  (e == 0 ? Z.u1y : Z.u2y)[og] = u[1];
  (e == 0 ? Z.u1z : Z.u2z)[og] = u[2];
  const double f = fjac * am;
  const double jac = 0.25 * fabs(f * f * f);
  double di[3], dk[3];
  const double ri = centre_offset(B, i, u, di), rk = centre_offset(B, k, u, dk);
  const double so = u_orb(B.n_sto[i], B.g_slater[i], ri), go = u_gauss(B, i, ri);
  const double so2 = same ? so : u_orb(B.n_sto[k], B.g_slater[k], rk);
  const double go2 = same ? go : u_gauss(B, k, rk);
  if (MODE != SS_PREC_FP64) (e == 0 ? Z.j1 : Z.j2)[og] = jac;
  const double ip = e == 0 ? 1.0 : 1.0 / pi0[s];
  for (int x = P.first[g]; x < P.first[g + 1]; x++) {
    const int p = P.order[x];
    const double poly_ik = poly(B, P.pi[p], di) * poly(B, P.pk[p], dk);
    double rs = poly_ik * so * so2, rg = poly_ik * go * go2;
    if (MODE == SS_PREC_FP64) {
      rs = jac * rs;
      rg = jac * rg;
      if (e == 1) {
        rs = rs * ip;
        rg = rg * ip;
      }
    }
    const int64_t o = (int64_t)p * Z.ld + s;
    (e == 0 ? Z.a_s : Z.b_s)[o] = rs;
    (e == 0 ? Z.a_g : Z.b_g)[o] = rg;
  }
}

// Accumulation (src/two_e_slater.F90:424-453).  One warp per (tile of quartets, walker slice); lanes
// stride over the walkers, so every quartet's partial sums have a fixed order.
//
// The FP64 pipe bounds it (two lanes per clock and SM).  A quartet and walker on their own cost it
// about 20 operations, 16 of them r12 and its inverse root; these are the same for all quartets of a
// tile, and the products with them for its quartets of one ket (FP64) or bra pair (REF32).  The
// 26-function water's 61,776 quartets make 6,250 tiles: 4 operations each.  16,000 walkers:
// 54 -> 13 ms (a warp per quartet before); the order of every sum is unchanged.
template <int MODE>
__global__ void __launch_bounds__(128, 2) zv_accum_kernel(int64_t S, ZvTiles Q, int nsplit, ZvChunk Z,
                                                          const double* __restrict__ pi0,
                                                          double* __restrict__ partS,
                                                          double* __restrict__ partG) {
  const int64_t item = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31, sp = (int)(item % nsplit);
  if (item / nsplit >= Q.n) return;
  const ZvTile& T = Q.tile[item / nsplit];
  const int64_t per = (S + nsplit - 1) / nsplit;
  const int64_t w0 = sp * per, w1 = min(S, w0 + per);
  const int64_t g1 = (int64_t)T.g1 * Z.ld, g2 = (int64_t)T.g2 * Z.ld;
  const uint64_t mask = T.mask;
  double sS[ZV_TB][ZV_TK], sG[ZV_TB][ZV_TK];
  int bra[ZV_TB], ket[ZV_TK];
#pragma unroll
  for (int t = 0; t < ZV_TB; t++) bra[t] = T.bra[t];
#pragma unroll
  for (int u = 0; u < ZV_TK; u++) ket[u] = T.ket[u];
#pragma unroll
  for (int t = 0; t < ZV_TB; t++)
#pragma unroll
    for (int u = 0; u < ZV_TK; u++) sS[t][u] = sG[t][u] = 0.0;
  for (int64_t s = w0 + lane; s < w1; s += 32) {
    const double dx = Z.u1x[g1 + s] - Z.u2x[g2 + s];
    const double dy = Z.u1y[g1 + s] - Z.u2y[g2 + s];
    const double dz = Z.u1z[g1 + s] - Z.u2z[g2 + s];
    const double r12_2 = dx * dx + dy * dy + dz * dz;
    double inv, factor = 1.0;
    if (MODE == SS_PREC_FP64) {
      inv = rsqrt(r12_2);
    } else {
      const double rj = Z.j1[g1 + s] * Z.j2[g2 + s];
      factor = (double)(__fdiv_rn((float)rj, (float)pi0[s]));
      inv = (double)(__fdiv_rn(1.0f, __fsqrt_rn((float)r12_2)));
    }
    double aS[ZV_TB], aG[ZV_TB];
#pragma unroll
    for (int t = 0; t < ZV_TB; t++) {
      aS[t] = aG[t] = 0.0;
      if (bra[t] >= 0) {
        aS[t] = Z.a_s[(int64_t)bra[t] * Z.ld + s];
        aG[t] = Z.a_g[(int64_t)bra[t] * Z.ld + s];
        if (MODE != SS_PREC_FP64) {
          aS[t] = factor * aS[t];
          aG[t] = factor * aG[t];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < ZV_TK; u++) {
      if (ket[u] < 0) continue;
      double bS = Z.b_s[(int64_t)ket[u] * Z.ld + s], bG = Z.b_g[(int64_t)ket[u] * Z.ld + s];
      if (MODE == SS_PREC_FP64) {
        bS = bS * inv;
        bG = bG * inv;
      }
#pragma unroll
      for (int t = 0; t < ZV_TB; t++) {
        if (!(mask >> (t * ZV_TK + u) & 1)) continue;
        if (MODE == SS_PREC_FP64) {
          sS[t][u] = fma(aS[t], bS, sS[t][u]);
          sG[t][u] = fma(aG[t], bG, sG[t][u]);
        } else {
          sS[t][u] = sS[t][u] + aS[t] * bS * inv;
          sG[t][u] = sG[t][u] + aG[t] * bG * inv;
        }
      }
    }
  }
  const int64_t* q = Q.q + T.q;
#pragma unroll
  for (int t = 0; t < ZV_TB; t++)
#pragma unroll
    for (int u = 0; u < ZV_TK; u++) {
      if (!(mask >> (t * ZV_TK + u) & 1)) continue;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sS[t][u] += __shfl_down_sync(0xffffffffu, sS[t][u], o);
        sG[t][u] += __shfl_down_sync(0xffffffffu, sG[t][u], o);
      }
      if (lane == 0) {
        partS[*q * nsplit + sp] = sS[t][u];
        partG[*q * nsplit + sp] = sG[t][u];
      }
      q++;
    }
}

__global__ void zv_reduce_partials(int64_t nint, int nsplit, const double* __restrict__ partS,
                                   const double* __restrict__ partG, double* __restrict__ eS,
                                   double* __restrict__ eG) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nint) return;
  double a = 0.0, g = 0.0;
  for (int t = 0; t < nsplit; t++) {
    a += partS[q * nsplit + t];
    g += partG[q * nsplit + t];
  }
  eS[q] += a;
  eG[q] += g;
}

// block moments (src/two_e_slater.F90:463-481)
__global__ void zv_block_stats(int64_t nint, int64_t npts, double* __restrict__ eS, double* __restrict__ eG,
                               double* __restrict__ acc, double* __restrict__ acc2) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nint) return;
  const double factor = 1.0 / (double)npts;
  const double x = eS[q] * factor - eG[q] * factor;
  acc[q] += x;
  acc2[q] += x * x;
  eS[q] = 0.0;
  eG[q] = 0.0;
}

// mean and error (src/two_e_slater.F90:488-492); unbiased=1 uses sqrt(var/(nb-1))
__global__ void zv_final(int64_t nint, int nb, int unbiased, const double* __restrict__ acc,
                         const double* __restrict__ acc2, double* __restrict__ mean,
                         double* __restrict__ sigma, unsigned long long* __restrict__ max_sigma_bits) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nint) return;
  const double m = acc[q] / nb, m2 = acc2[q] / nb;
  double e;
  if (unbiased)
    e = nb > 1 ? sqrt(fabs(m2 - m * m) / (double)(nb - 1)) : 0.0;
  else
    e = sqrt(fabs(m2 - m * m)) / sqrt((double)nb);
  mean[q] = m;
  sigma[q] = e;
  if (max_sigma_bits) atomicMax(max_sigma_bits, (unsigned long long)__double_as_longlong(e));
}

// ---------------------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------------------
cudaError_t launch_draw_walkers(cudaStream_t st, uint64_t seed, int64_t first, int64_t S, double* r1,
                                double* r2) {
  if (S <= 0) return cudaSuccess;
  draw_walkers_kernel<<<(unsigned)((S + 255) / 256), 256, 0, st>>>(seed, first, S, r1, r2);
  return cudaGetLastError();
}

cudaError_t launch_walker_aux(cudaStream_t st, int64_t S, const double* r1, const double* r2, double* r1m,
                              double* r2m, double* pi0) {
  if (S <= 0) return cudaSuccess;
  walker_aux_kernel<<<(unsigned)((S + 255) / 256), 256, 0, st>>>(S, r1, r2, r1m, r2m, pi0);
  return cudaGetLastError();
}

cudaError_t launch_zv_pairs(cudaStream_t st, int mode, const BasisDev& B, const ZvPairs& P,
                            int64_t S, const double* r1, const double* r2, const double* r1m,
                            const double* r2m, const double* pi0, const ZvChunk& Z) {
  dim3 grid((unsigned)((S + 127) / 128), (unsigned)P.ngroups, 2);
  if (mode == SS_PREC_FP64)
    zv_pair_kernel<SS_PREC_FP64><<<grid, 128, 0, st>>>(B, P, S, r1, r2, r1m, r2m, pi0, Z);
  else
    zv_pair_kernel<SS_PREC_REF32><<<grid, 128, 0, st>>>(B, P, S, r1, r2, r1m, r2m, pi0, Z);
  return cudaGetLastError();
}

cudaError_t launch_zv_accum(cudaStream_t st, int mode, int nsplit, int64_t S, const ZvTiles& Q,
                            const ZvChunk& Z, const double* pi0, double* partS, double* partG) {
  if (Q.n <= 0) return cudaSuccess;
  dim3 grid((unsigned)(((int64_t)Q.n * nsplit + 3) / 4));
  if (mode == SS_PREC_FP64)
    zv_accum_kernel<SS_PREC_FP64><<<grid, 128, 0, st>>>(S, Q, nsplit, Z, pi0, partS, partG);
  else
    zv_accum_kernel<SS_PREC_REF32><<<grid, 128, 0, st>>>(S, Q, nsplit, Z, pi0, partS, partG);
  return cudaGetLastError();
}

cudaError_t launch_zv_reduce(cudaStream_t st, int64_t nint, int nsplit, const double* partS,
                             const double* partG, double* eS, double* eG) {
  zv_reduce_partials<<<(unsigned)((nint + 255) / 256), 256, 0, st>>>(nint, nsplit, partS, partG, eS, eG);
  return cudaGetLastError();
}

cudaError_t launch_zv_block_stats(cudaStream_t st, int64_t nint, int64_t npts, double* eS, double* eG,
                                  double* acc, double* acc2) {
  zv_block_stats<<<(unsigned)((nint + 255) / 256), 256, 0, st>>>(nint, npts, eS, eG, acc, acc2);
  return cudaGetLastError();
}

cudaError_t launch_zv_final(cudaStream_t st, int64_t nint, int nb, int unbiased, const double* acc,
                            const double* acc2, double* mean, double* sigma, unsigned long long* maxbits) {
  zv_final<<<(unsigned)((nint + 255) / 256), 256, 0, st>>>(nint, nb, unbiased, acc, acc2, mean, sigma,
                                                           maxbits);
  return cudaGetLastError();
}

}  // namespace ss
