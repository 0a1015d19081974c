// one_e.cu -- one-electron integrals of the STO Gaussian fits: overlap S, nuclear attraction V
// and kinetic K for every function pair (i,k), as the reference's one_e_slater program computes
// them (src/one_e_slater.F90:81-89, src/one_elect.F90:1-105).
//
// One CTA per function pair i >= k (the operators are symmetric: (k,i) is the same value); its
// threads share the items (m1, m2, nucleus) and the block sums them in a fixed order, so results
// are run-to-run deterministic.  Per item:
//  * S: exp(-mu |A-B|^2) Ix Iy Iz, the one-dimensional overlaps by s(a+1,c) = (P-A) s(a,c) +
//    (a s(a-1,c) + c s(a,c-1)) / 2p, skipped where mu |A-B|^2 > -ln(1e-15) as the reference
//    (src/one_electron_sij.F90, src/one_electron_I.F90);
//  * K: the reference's three overlap terms (src/one_electron_Kij.F90) from the same table;
//  * V: -sum_C Z_C NAI(A,B,C) (src/one_electron_Vij.F90, src/NAI_pol_mult.F90): per axis the
//    polynomial in u = t^2 of I_x1_pol_mult_mono_elec, built bottom-up in the recursion's order
//      I(0,c) = (c-1) R2 I(0,c-2) + R1' I(0,c-1),  I(1,c) = c R2 I(0,c-1) + R1 I(0,c),
//      I(a,c) = (a-1) R2 I(a-2,c) + c R2 I(a-1,c-1) + R1 I(a-1,c)
//    with R1 = (P-A) - (P-C) u, R1' = (P-B) - (P-C) u, R2 = (1 - u)/(2p), then the product of the
//    three axes and sum_i d(i) F_i(p |P-C|^2), coefficients below 1e-9 skipped as in NAI_pol_mult.
// The exponentials and the Boys function of an item serve all cartesian components of the r^2-type
// fits, and every table has compile-time bounds (powers <= 2 per function and axis, which
// ss_basis_set guarantees), so it stays in registers.  With the tables indexed at run time they
// lived in local memory: 26.1 ms for the 26-function water (20 Gaussians), 0.64 ms now.
#include <math.h>

#include <algorithm>

#include "boys.cuh"
#include "ss_common.cuh"
#include "ss_context.cuh"

namespace ss {

constexpr int OE_MAXP = 2;  // power of one function on one axis, incl. the +2 of r^2 fits
constexpr int OE_NF = 8;    // Boys orders: total power of the pair <= 8

// out += (r0 + r1 u) b, b of degree deg
template <int DEG>
__device__ __forceinline__ void oe_mul_add(const double (&b)[5], double r0, double r1, double (&out)[5]) {
#pragma unroll
  for (int m = 0; m <= DEG; m++) {
    out[m] = fma(r0, b[m], out[m]);
    if (m + 1 < 5) out[m + 1 < 5 ? m + 1 : 4] = fma(r1, b[m], out[m + 1 < 5 ? m + 1 : 4]);
  }
}

// one entry of the table, with the recursion of I_x1_pol_mult_mono_elec
template <int A, int C>
__device__ __forceinline__ void oe_entry(double (&I)[3][3][5], double pa, double pb, double pc, double h) {
  double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if constexpr (A == 0 && C == 0) {
    v[0] = 1.0;
  } else if constexpr (A == 0) {
    if constexpr (C >= 2) oe_mul_add<C - 2>(I[0][C - 2], (C - 1) * h, -((C - 1) * h), v);
    oe_mul_add<C - 1>(I[0][C - 1], pb, -pc, v);
  } else {
    if constexpr (A >= 2) oe_mul_add<A - 2 + C>(I[A - 2][C], (A - 1) * h, -((A - 1) * h), v);
    if constexpr (C >= 1) oe_mul_add<A + C - 2>(I[A - 1][C - 1], C * h, -(C * h), v);
    oe_mul_add<A - 1 + C>(I[A - 1][C], pa, -pc, v);
  }
#pragma unroll
  for (int m = 0; m < 5; m++) I[A][C][m] = v[m];
}

// per-axis polynomial I(a,c)(u); a, c are uniform over the CTA
__device__ __forceinline__ void oe_axis(int a, int c, double pa, double pb, double pc, double h, double (&out)[5]) {
  double I[3][3][5];
  oe_entry<0, 0>(I, pa, pb, pc, h);
  oe_entry<0, 1>(I, pa, pb, pc, h);
  oe_entry<0, 2>(I, pa, pb, pc, h);
  oe_entry<1, 0>(I, pa, pb, pc, h);
  oe_entry<1, 1>(I, pa, pb, pc, h);
  oe_entry<1, 2>(I, pa, pb, pc, h);
  oe_entry<2, 0>(I, pa, pb, pc, h);
  oe_entry<2, 1>(I, pa, pb, pc, h);
  oe_entry<2, 2>(I, pa, pb, pc, h);
#pragma unroll
  for (int m = 0; m < 5; m++) out[m] = 0.0;
#pragma unroll
  for (int x = 0; x < 3; x++)
#pragma unroll
    for (int y = 0; y < 3; y++)
      if (x == a && y == c) {
#pragma unroll
        for (int m = 0; m < 5; m++) out[m] = I[x][y][m];
      }
}

// one-dimensional overlaps of powers (a', c), a' = a - 2, a, a + 2 (0 where a' < 0), without sqrt(pi/p)
__device__ __forceinline__ void oe_overlap(int a, int c, double pa, double pb, double h, double& lo, double& mid,
                                           double& hi) {
  double s[5][3];
#pragma unroll
  for (int y = 0; y < 3; y++)
#pragma unroll
    for (int x = 0; x < 5; x++) {
      double v;
      if (x == 0 && y == 0) {
        v = 1.0;
      } else if (x > 0) {
        v = pa * s[x - 1][y];
        if (x > 1) v = fma((x - 1) * h, s[x > 1 ? x - 2 : 0][y], v);
        if (y > 0) v = fma(y * h, s[x - 1][y > 0 ? y - 1 : 0], v);
      } else {
        v = pb * s[0][y > 0 ? y - 1 : 0];
        if (y > 1) v = fma((y - 1) * h, s[0][y > 1 ? y - 2 : 0], v);
      }
      s[x][y] = v;
    }
  lo = mid = hi = 0.0;
#pragma unroll
  for (int x = 0; x < 3; x++)
#pragma unroll
    for (int y = 0; y < 3; y++)
      if (x == a && y == c) {
        mid = s[x][y];
        hi = s[x + 2][y];
        lo = x >= 2 ? s[x >= 2 ? x - 2 : 0][y] : 0.0;
      }
}

__global__ void __launch_bounds__(128) one_e_kernel(BasisDev B, int nat, const double* __restrict__ xyz,
                                                    const double* __restrict__ charge, double* __restrict__ S,
                                                    double* __restrict__ V, double* __restrict__ K) {
  __shared__ double s_boys[BOYS_SMEM_DOUBLES];
  __shared__ double s_red[3][4];
  boys_tables_to_smem(s_boys);
  __syncthreads();
  const int n = B.n;
  int i = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
  while ((int64_t)i * (i + 1) / 2 > blockIdx.x) i--;
  while ((int64_t)(i + 1) * (i + 2) / 2 <= blockIdx.x) i++;
  const int k = (int)(blockIdx.x - (int64_t)i * (i + 1) / 2);
  const int ti = B.i_type[i] == 2, tk = B.i_type[k] == 2;
  const int ni = ti ? 3 : 1, nk = tk ? 3 : 1;
  int pi[3], pk[3], tot = 2 * (ti + tk);
#pragma unroll
  for (int l = 0; l < 3; l++) {
    pi[l] = B.npower[3 * i + l];
    pk[l] = B.npower[3 * k + l];
    tot += pi[l] + pk[l];
  }
  const double A[3] = {B.center[3 * i], B.center[3 * i + 1], B.center[3 * i + 2]};
  const double C[3] = {B.center[3 * k], B.center[3 * k + 1], B.center[3 * k + 2]};
  double dist = 0.0;
#pragma unroll
  for (int l = 0; l < 3; l++) dist = dist + (A[l] - C[l]) * (A[l] - C[l]);
  const int ngk = B.n_gauss[k], np = B.n_gauss[i] * ngk;
  const double pi_ = 3.14159265358979323846;
  double s = 0.0, v = 0.0, kin = 0.0;
  const int per = nat > 0 ? nat : 1;
  for (int e = threadIdx.x; e < np * per; e += blockDim.x) {
    const int kn = e / np, m = e - kn * np;
    const int m1 = m / ngk, m2 = m - m1 * ngk;
    const double ga = B.g_gauss[m1 + (int64_t)B.ld * i], gb = B.g_gauss[m2 + (int64_t)B.ld * k];
    const double dd = B.c_gauss[m1 + (int64_t)B.ld * (i + (int64_t)n * ti)] *
                      B.c_gauss[m2 + (int64_t)B.ld * (k + (int64_t)n * tk)];
    const double p = ga + gb, p_inv = 1.0 / p, h = 0.5 * p_inv, rho = ga * gb * p_inv;
    const double ex = exp(-(dist * rho));
    double P[3], PA[3], PB[3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
      P[l] = (ga * A[l] + gb * C[l]) * p_inv;
      PA[l] = P[l] - A[l];
      PB[l] = P[l] - C[l];
    }
    if (kn == 0 && !(rho * dist > 34.538776394910684)) {  // -ln(1e-15)
      const double w = dd * ex * (sqrt(pi_ * p_inv) * (pi_ * p_inv));
      for (int x = 0; x < ni; x++)
        for (int y = 0; y < nk; y++) {
          double lo[3], mid[3], hi[3];
          int a[3], na = 0;
#pragma unroll
          for (int l = 0; l < 3; l++) {
            a[l] = pi[l] + ((ti && l == x) ? 2 : 0);
            na += a[l];
            oe_overlap(a[l], pk[l] + ((tk && l == y) ? 2 : 0), PA[l], PB[l], h, lo[l], mid[l], hi[l]);
          }
          const double sab = mid[0] * mid[1] * mid[2];
          const double up = hi[0] * mid[1] * mid[2] + mid[0] * hi[1] * mid[2] + mid[0] * mid[1] * hi[2];
          const double dn = (double)(a[0] * (a[0] - 1)) * lo[0] * mid[1] * mid[2] +
                            (double)(a[1] * (a[1] - 1)) * mid[0] * lo[1] * mid[2] +
                            (double)(a[2] * (a[2] - 1)) * mid[0] * mid[1] * lo[2];
          s += w * sab;
          kin += w * (ga * (3.0 + 2.0 * na) * sab - 2.0 * ga * ga * up - 0.5 * dn);
        }
    }
    if (nat > 0) {
      double PC[3], r2 = 0.0;
#pragma unroll
      for (int l = 0; l < 3; l++) {
        PC[l] = P[l] - xyz[3 * kn + l];
        r2 = r2 + PC[l] * PC[l];
      }
      double F[OE_NF + 1];
      boys_tab<OE_NF>(p * r2, tot, F, s_boys);
      double nai = 0.0;
      for (int x = 0; x < ni; x++)
        for (int y = 0; y < nk; y++) {
          double d[OE_NF + 1];
#pragma unroll
          for (int t = 0; t <= OE_NF; t++) d[t] = 0.0;
          d[0] = 1.0;
          if (tot > 0) {
            double X[5], Y[5], Z[5], xy[9];
            oe_axis(pi[0] + ((ti && x == 0) ? 2 : 0), pk[0] + ((tk && y == 0) ? 2 : 0), PA[0], PB[0], PC[0], h, X);
            oe_axis(pi[1] + ((ti && x == 1) ? 2 : 0), pk[1] + ((tk && y == 1) ? 2 : 0), PA[1], PB[1], PC[1], h, Y);
            oe_axis(pi[2] + ((ti && x == 2) ? 2 : 0), pk[2] + ((tk && y == 2) ? 2 : 0), PA[2], PB[2], PC[2], h, Z);
#pragma unroll
            for (int t = 0; t < 9; t++) xy[t] = 0.0;
#pragma unroll
            for (int u = 0; u < 5; u++)
#pragma unroll
              for (int w = 0; w < 5; w++) xy[u + w] = fma(X[u], Y[w], xy[u + w]);
            d[0] = 0.0;
#pragma unroll
            for (int u = 0; u < 9; u++)
#pragma unroll
              for (int w = 0; w < 5; w++)
                if (u + w <= OE_NF) d[u + w] = fma(xy[u], Z[w], d[u + w]);
          }
#pragma unroll
          for (int t = 0; t <= OE_NF; t++)
            if (t <= tot && !(fabs(d[t]) < 1.e-9)) nai = fma(d[t], F[t], nai);
        }
      v -= charge[kn] * dd * (2.0 * pi_ * ex * p_inv) * nai;
    }
  }
  double vals[3] = {s, v, kin};
#pragma unroll
  for (int t = 0; t < 3; t++) {
    double x = vals[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) s_red[t][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    const int64_t o = threadIdx.x == 0 ? i + (int64_t)n * k : k + (int64_t)n * i;
    S[o] = ((s_red[0][0] + s_red[0][1]) + s_red[0][2]) + s_red[0][3];
    V[o] = ((s_red[1][0] + s_red[1][1]) + s_red[1][2]) + s_red[1][3];
    K[o] = ((s_red[2][0] + s_red[2][1]) + s_red[2][2]) + s_red[2][3];
  }
}

int pool_get(ss_ctx* c, const char* name, size_t bytes, void** out);

}  // namespace ss

using namespace ss;

extern "C" {

int ss_nuclei_set(ss_ctx* c, int nat, const double* xyz, const double* charge) {
  if (!c) {
    ss_set_error_msg("null context");
    return SS_ERR_ARG;
  }
  if (nat < 0 || (nat > 0 && (!xyz || !charge))) {
    ss_set_error_msg("ss_nuclei_set: bad arguments (nat=%d)", nat);
    return SS_ERR_ARG;
  }
  c->h_nuc_xyz.assign(xyz, xyz + 3 * (size_t)nat);
  c->h_nuc_charge.assign(charge, charge + (size_t)nat);
  return SS_OK;
}

int ss_one_e(ss_ctx* c, double* S, double* V, double* K) {
  if (!c) {
    ss_set_error_msg("null context");
    return SS_ERR_ARG;
  }
  SS_CUDA_TRY(cudaSetDevice(c->device));
  if (!c->n) {
    ss_set_error_msg("ss_one_e needs ss_basis_set first");
    return SS_ERR_STATE;
  }
  for (int f = 0; f < c->n; f++) {
    int tot = c->h_itype[f] == 1 ? 0 : 2;
    for (int ax = 0; ax < 3; ax++) {
      tot += c->h_npower[3 * f + ax];
      if (c->h_npower[3 * f + ax] + (c->h_itype[f] == 1 ? 0 : 2) > OE_MAXP) {
        ss_set_error_msg("ss_one_e: function %d has a per-axis power above %d", f + 1, OE_MAXP);
        return SS_ERR_UNSUPPORTED;
      }
    }
    if (2 * tot > OE_NF) {
      ss_set_error_msg("ss_one_e: function %d has a total power above %d", f + 1, OE_NF / 2);
      return SS_ERR_UNSUPPORTED;
    }
  }
  const int n = c->n, nat = (int)c->h_nuc_charge.size();
  const size_t nn = (size_t)n * n;
  void *p_xyz, *p_ch, *p_out;
  int rc = pool_get(c, "oe_xyz", sizeof(double) * std::max<size_t>(3 * (size_t)nat, 1), &p_xyz);
  if (!rc) rc = pool_get(c, "oe_charge", sizeof(double) * std::max<size_t>((size_t)nat, 1), &p_ch);
  if (!rc) rc = pool_get(c, "oe_out", sizeof(double) * 3 * nn, &p_out);
  if (rc) return rc;
  if (nat) {
    SS_CUDA_TRY(cudaMemcpyAsync(p_xyz, c->h_nuc_xyz.data(), sizeof(double) * 3 * nat, cudaMemcpyHostToDevice,
                                c->stream));
    SS_CUDA_TRY(cudaMemcpyAsync(p_ch, c->h_nuc_charge.data(), sizeof(double) * nat, cudaMemcpyHostToDevice,
                                c->stream));
  }
  double* out = (double*)p_out;
  one_e_kernel<<<(unsigned)((size_t)n * (n + 1) / 2), 128, 0, c->stream>>>(c->basis, nat, (const double*)p_xyz, (const double*)p_ch, out,
                                                     out + nn, out + 2 * nn);
  SS_CUDA_TRY(cudaGetLastError());
  c->launches++;
  if (S) SS_CUDA_TRY(cudaMemcpyAsync(S, out, sizeof(double) * nn, cudaMemcpyDeviceToHost, c->stream));
  if (V) SS_CUDA_TRY(cudaMemcpyAsync(V, out + nn, sizeof(double) * nn, cudaMemcpyDeviceToHost, c->stream));
  if (K) SS_CUDA_TRY(cudaMemcpyAsync(K, out + 2 * nn, sizeof(double) * nn, cudaMemcpyDeviceToHost, c->stream));
  SS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return SS_OK;
}

}  // extern "C"
