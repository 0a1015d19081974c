// shell_lane.cuh -- the two-float and FP32 tiers of light shell quartets: one bra primitive per
// lane (instantiated per ket type in shell_lane_*.cu).
//
// shell_eri.cuh passes the Hermite integrals through shared memory, with barriers, segments and
// index arithmetic around them.  With the work off the FP64 pipe that overhead was most of the
// instructions (3,100 per 32 primitive quartets of the 26-function water, 40 % of the issue slots
// used).  Here a lane keeps its bra primitive, the Hermite integrals and its sums over the kets
// G[t][f] in registers; all lanes of a warp take the same ket, so the ket's record and its
// coefficients are broadcasts from shared memory, and every index is known at compile time.  The
// bra's coefficients are applied once per lane and CTA, at the end.
//
// What bounds it: the issue rate of the FP32 pipe (a two-float multiply-add is 12 instructions) and
// the registers, which set how many components of the ket a pass can hold (sh_lane_chunk); a chunk
// repeats the Hermite integrals.  Heavier classes (sh_lane_chunk = 0) stay with shell_eri.cuh,
// which shares the integrals among all components.  The FP64 tier of every class does too: it is
// a tenth of the work and runs beside these kernels on the other pipe.
#pragma once
#include "shell_eri.cuh"

namespace ss {

#ifdef __CUDACC__

// compile-time description of a ket type: terms of the components [F0, F0 + NF)
template <int TA, int TB, bool SAME, bool ONEC>
struct LaneKet {
  static constexpr ShStruct S = sh_struct(TA, TB, SAME, ONEC);
};

template <typename Real>
__device__ __forceinline__ Real lane_zero();
template <>
__device__ __forceinline__ df lane_zero<df>() { return df{0.f, 0.f}; }
template <>
__device__ __forceinline__ float lane_zero<float>() { return 0.f; }

// powers of k / s_P and k / s_Q (shell_eri.cuh) of an item
struct LaneUnit {
  float a[5], b[5];
};
__device__ __forceinline__ df r_scale(df x, float k) { return df_scale(x, k); }
__device__ __forceinline__ float r_scale(float x, float k) { return x * k; }

// G[f][t] += R[t + tau] e (k / s_P)^|t| (k / s_Q)^|tau| for all bra Hermite functions t (ONE4: only where
// t + tau is even on every axis)
template <uint32_t TAU, bool ONE4, typename Real, int NR, int H, int... T>
__device__ __forceinline__ void lane_term(const Real (&R)[NR], Real e, const LaneUnit& u, Real (&G)[H],
                                          std::integer_sequence<int, T...>) {
  constexpr int dtau = (int)((TAU & 255) + ((TAU >> 8) & 255) + (TAU >> 16));
  Real ed[5];  // by the degree of t
  ed[0] = dtau ? r_scale(e, u.b[dtau]) : e;
#pragma unroll
  for (int d = 1; d < 5; d++)
    if (H >= sh_nherm(d)) ed[d] = r_scale(ed[0], u.a[d]);
  auto one = [&](auto tc) {
    constexpr int t = decltype(tc)::value;
    constexpr ShDeg h = sh_degs(t);
    constexpr int x = h.t + (int)(TAU & 255), y = h.u + (int)((TAU >> 8) & 255), z = h.v + (int)(TAU >> 16);
    if constexpr (!ONE4 || !((x | y | z) & 1)) G[t] = r_fma(R[sh_hidx(x, y, z)], ed[h.t + h.u + h.v], G[t]);
  };
  (one(std::integral_constant<int, T>()), ...);
}
__device__ __forceinline__ df lane_load(const float2* e, df) {
  const float2 v = *e;
  return df{v.x, v.y};
}
__device__ __forceinline__ float lane_load(const float2* e, float) { return e->x; }

template <class KET, int X, int X1, bool ONE4, typename Real, int NR, int H>
__device__ __forceinline__ void lane_comp(const Real (&R)[NR], const float2* e, const LaneUnit& u, Real (&G)[H]) {
  if constexpr (X < X1) {
    lane_term<KET::S.term[X], ONE4>(R, lane_load(e + X, Real()), u, G, std::make_integer_sequence<int, H>());
    lane_comp<KET, X + 1, X1, ONE4>(R, e, u, G);
  }
}
template <class KET, int F0, int F, int NF, bool ONE4, typename Real, int NR, int H>
__device__ __forceinline__ void lane_comps(const Real (&R)[NR], const float2* e, const LaneUnit& u, Real (&G)[NF][H]) {
  if constexpr (F < NF) {
    lane_comp<KET, KET::S.fs[F0 + F], KET::S.fs[F0 + F + 1], ONE4>(R, e, u, G[F]);
    lane_comps<KET, F0, F + 1, NF, ONE4>(R, e, u, G);
  }
}

// Hermite integrals of one primitive quartet in registers
template <int L, bool ONE4>
__device__ __forceinline__ void lane_hermite(const ShPrimF& a, const ShPrimF& b, float kx, float ik2,
                                             const float* boys, df (&R)[sh_nherm(L)]) {
  const df pa{a.p[0], a.p[1]}, pb{b.p[0], b.p[1]};
  const df rs = df_rsqrt(df_add(pa, pb));
  const df pre = df_mul(df_mul(df{a.w[0], a.w[1]}, df{b.w[0], b.w[1]}), rs);
  const df alpha = df_mul(df_mul(pa, rs), df_mul(pb, rs));
  const df m2a = df_scale(alpha, -2.f * ik2);
  df bs[L + 1];
  if constexpr (ONE4) {
    bs[0] = pre;
    df pw = pre;
#pragma unroll
    for (int m = 1; m <= L; m++) {
      const float ih = 1.f / (2 * m + 1);
      pw = df_mul(pw, m2a);
      bs[m] = df_mul(pw, df{ih, (float)(1.0 / (2 * m + 1) - (double)ih)});
    }
    store_row_1c<L, df>(bs, R);
  } else {
    const df X = sh_distance(a, b, 0), Y = sh_distance(a, b, 1), Z = sh_distance(a, b, 2);
    df F[L + 1];
    boys_shell<L>(df_renorm(df_mul(alpha, df_fma(X, X, df_fma(Y, Y, df_mul(Z, Z))))), F, boys);
    df pw = pre;
#pragma unroll
    for (int m = 0; m <= L; m++) {
      bs[m] = df_mul(pw, F[m]);
      if (m < L) pw = df_mul(pw, m2a);
    }
    R[0] = bs[L];
    hermite_levels<L, L - 1>(df_scale(X, kx), df_scale(Y, kx), df_scale(Z, kx), bs, R);
  }
}
template <int L, bool ONE4>
__device__ __forceinline__ void lane_hermite(const ShPrimF& a, const ShPrimF& b, float kx, float ik2,
                                             const float* boys, float (&R)[sh_nherm(L)]) {
  const float rs = rsqrtf(a.p[0] + b.p[0]);
  const float pre = a.w[0] * b.w[0] * rs;
  const float alpha = (a.p[0] * rs) * (b.p[0] * rs);
  const float m2a = -2.f * (alpha * ik2);
  float bs[L + 1];
  if constexpr (ONE4) {
    bs[0] = pre;
    float pw = pre;
#pragma unroll
    for (int m = 1; m <= L; m++) {
      pw *= m2a;
      bs[m] = pw * (1.f / (2 * m + 1));
    }
    store_row_1c<L, float>(bs, R);
  } else {
    const float X = (a.ph[0] - b.ph[0]) + (a.pl[0] - b.pl[0]);
    const float Y = (a.ph[1] - b.ph[1]) + (a.pl[1] - b.pl[1]);
    const float Z = (a.ph[2] - b.ph[2]) + (a.pl[2] - b.pl[2]);
    float F[L + 1];
    boys_shell<L>(alpha * fmaf(X, X, fmaf(Y, Y, Z * Z)), F, boys);
    float pw = pre;
#pragma unroll
    for (int m = 0; m <= L; m++) {
      bs[m] = pw * F[m];
      if (m < L) pw *= m2a;
    }
    R[0] = bs[L];
    hermite_levels<L, L - 1>(X * kx, Y * kx, Z * kx, bs, R);
  }
}

// the warp's kets of a tier: the union of its lanes' ranges [lo, hi)
__device__ __forceinline__ void lane_range(int lo, int hi, int& qa, int& qb) {
  qa = hi > lo ? lo : 1 << 30;
  qb = hi > lo ? hi : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    qa = min(qa, __shfl_xor_sync(0xffffffffu, qa, o));
    qb = max(qb, __shfl_xor_sync(0xffffffffu, qb, o));
  }
}

// one ket summed into G
template <typename Real, class KET, int DB, int F0, int NF, bool ONE4>
__device__ __forceinline__ void lane_ket(const ShPrimF& P, int q, const ShPrimF* s_ket, const float2* s_E,
                                         const float* boys, Real (&G)[NF][sh_nherm(DB)]) {
  constexpr int L = DB + KET::S.d;
  const ShPrimF& Q = s_ket[q];
  const float kx = fminf(P.s, Q.s), ik = fmaxf(P.is, Q.is);
  Real R[sh_nherm(L)];
  lane_hermite<L, ONE4>(P, Q, kx, ik * ik, boys, R);
  LaneUnit u;
  u.a[1] = kx * P.is;
  u.b[1] = kx * Q.is;
#pragma unroll
  for (int d = 2; d < 5; d++) {
    u.a[d] = u.a[d - 1] * u.a[1];
    u.b[d] = u.b[d - 1] * u.b[1];
  }
  lane_comps<KET, F0, 0, NF, ONE4>(R, s_E + q * KET::S.nterm, u, G);
}

template <class KET, int DB>
struct LaneDim {
  static constexpr int H = sh_nherm(DB), L = DB + KET::S.d;
  static constexpr int MINB = L >= 4 || H >= 10 ? 2 : 3;
  // shared memory: Boys table, ket records and coefficients, then the sums G of the four warps in
  // the place of the ket's
  static constexpr int KETS = sh_lane_kets(L);
  static constexpr size_t ket_bytes = KETS * (sizeof(ShPrimF) + sizeof(float2) * KET::S.nterm);
};

template <class KET, int DB, int F0, int NF, bool ONE4>
__device__ __forceinline__ void lane_body(const ShArgs& A, const ShWork& W, int blk, int kc, float* s_boys, char* s_mem,
                                          double (&s_red)[4][64]) {
  constexpr int H = sh_nherm(DB), L = DB + KET::S.d, NT = KET::S.nterm;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ShPair B = A.pair[W.bra], K = A.pair[W.ket];
  const int nb = A.cnt[W.bra], nk = A.cnt[W.ket];
  constexpr int KETS = LaneDim<KET, DB>::KETS;
  const int p0 = blk * SH_LANE_BRA, k0 = kc * KETS, k1 = min(nk, k0 + KETS);
  const int p = p0 + tid;
  ShPrimF* s_ket = reinterpret_cast<ShPrimF*>(s_mem);
  float2* s_E = reinterpret_cast<float2*>(s_ket + KETS);
  df* s_G = reinterpret_cast<df*>(s_mem) + warp * (H * NF * 33);  // [t * NF + f][lane], after the kets
  const ShPrim* bra = A.prim + B.prim_off;
  const ShPrim* ket = A.prim + K.prim_off;

  // ranges of this lane's kets in the chunk: [cd, cf) two floats, [cf, c) FP32
  int cd = k0, cf = k0, c = k0;
  if (p < nb && k1 > k0) {
    const double sb = bra[p].S;
    auto first_below = [&](double thr) {
      int lo = k0, hi = k1;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sb * ket[mid].S < thr) hi = mid; else lo = mid + 1;
      }
      return lo;
    };
    c = first_below(A.eps);
    cf = first_below(A.eps32);
    cd = first_below(A.eps_df);
  }
  df G[NF][H];
#pragma unroll
  for (int f = 0; f < NF; f++)
#pragma unroll
    for (int t = 0; t < H; t++) G[f][t] = lane_zero<df>();
  const bool any = __syncthreads_or(c > cd);
  if (any) {
    const float4* src = reinterpret_cast<const float4*>(A.boys[L].f);
    float4* dst = reinterpret_cast<float4*>(s_boys);
    for (int i = tid; i < SH_BOYS_K * SH_BOYS_ROW / 4; i += SH_LANE_BRA) dst[i] = src[i];
    const int n = k1 - k0;
    const float4* ksrc = reinterpret_cast<const float4*>(A.primf + K.prim_off + k0);
    float4* kdst = reinterpret_cast<float4*>(s_ket);
    for (int i = tid; i < n * (int)(sizeof(ShPrimF) / sizeof(float4)); i += SH_LANE_BRA) kdst[i] = ksrc[i];
    const float2* esrc = A.E2 + K.e_off + (size_t)k0 * NT;
    const ShStruct& SK = A.st[K.st];
    for (int i = tid; i < n * NT; i += SH_LANE_BRA) {
      const float sign = (sh_degree(SK.term[i % NT]) & 1) ? -1.f : 1.f;  // (-1)^|tau|
      const float2 e = esrc[i];
      s_E[i] = make_float2(e.x * sign, e.y * sign);
    }
    __syncthreads();
    ShPrimF P{};
    if (p < nb) P = A.primf[B.prim_off + p];
    // all lanes of a warp take the same ket; a lane outside its own range sits it out
    int qa, qb;
    lane_range(cd - k0, cf - k0, qa, qb);
    for (int q = qa; q < qb; q++)
      if (q >= cd - k0 && q < cf - k0) lane_ket<df, KET, DB, F0, NF, ONE4>(P, q, s_ket, s_E, s_boys, G);
    // FP32 sums of at most eight kets, then into the two-float sums
    lane_range(cf - k0, c - k0, qa, qb);
    for (int q8 = qa; q8 < qb; q8 += 8) {
      float Gf[NF][H];
#pragma unroll
      for (int f = 0; f < NF; f++)
#pragma unroll
        for (int t = 0; t < H; t++) Gf[f][t] = 0.f;
      for (int q = q8; q < min(q8 + 8, qb); q++)
        if (q >= cf - k0 && q < c - k0) lane_ket<float, KET, DB, F0, NF, ONE4>(P, q, s_ket, s_E, s_boys, Gf);
#pragma unroll
      for (int f = 0; f < NF; f++)
#pragma unroll
        for (int t = 0; t < H; t++) G[f][t] = df_add(G[f][t], df{Gf[f][t], 0.f});
    }
    __syncthreads();  // the kets' place becomes the sums'
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
      for (int t = 0; t < H; t++) s_G[(t * NF + f) * 33 + lane] = df_renorm(G[f][t]);
    __syncwarp();
  }
  // bra coefficients: lane <-> output (a, f), summed over the warp's 32 bra primitives
  const ShStruct& SB = A.st[B.st];
  const int nout = B.ncomp * NF, tot = W.split + W.lsplit, slot = W.split + blk * W.nkc + kc;
  const int np = min(32, nb - p0 - warp * 32);
  for (int o = lane; o < nout; o += 32) {
    df s{0.f, 0.f};
    if (any) {
      const int a = o / NF, f = o - a * NF;
      for (int x = SB.fs[a]; x < SB.fs[a + 1]; x++) {
        const uint32_t ht = SB.term[x];
        const df* g = s_G + (sh_pack_idx(ht) * NF + f) * 33;
        const float2* eb = A.E2 + B.e_off + (size_t)(p0 + warp * 32) * B.nterm + x;
        df v{0.f, 0.f};
        for (int i = 0; i < np; i++, eb += B.nterm) {
          const float2 e = *eb;
          v = df_fma(df{e.x, e.y}, g[i], v);
        }
        s = df_renorm(df_add(s, v));
      }
    }
    s_red[warp][o] = df_to(s);
  }
  __syncthreads();
  const double scale = SH_PI_5_2 * (A.scale[W.bra] * A.scale[W.ket]);
  for (int o = tid; o < nout; o += SH_LANE_BRA) {
    const int a = o / NF, f = o - a * NF;
    A.partial[W.part + (int64_t)(a * K.ncomp + F0 + f) * tot + slot] =
        scale * (((s_red[0][o] + s_red[1][o]) + s_red[2][o]) + s_red[3][o]);
  }
}

template <class KET, int DB, int F0, int NF, bool ONE4>
__device__ __forceinline__ void lane_chunk(int ch, const ShArgs& A, const ShWork& W, int blk, int kc, float* s_boys,
                                           char* s_mem, double (&s_red)[4][64]) {
  if constexpr (F0 < KET::S.ncomp) {
    if (ch == F0 / NF)
      lane_body<KET, DB, F0, (NF < KET::S.ncomp - F0 ? NF : KET::S.ncomp - F0), ONE4>(A, W, blk, kc, s_boys, s_mem, s_red);
    else
      lane_chunk<KET, DB, F0 + NF, NF, ONE4>(ch, A, W, blk, kc, s_boys, s_mem, s_red);
  }
}

template <class KET, int DB, int NF, bool ONE4>
__global__ void __launch_bounds__(SH_LANE_BRA, (LaneDim<KET, DB>::MINB)) shell_lane_kernel(ShArgs A) {
  extern __shared__ float4 sh_lane_raw[];
  float* s_boys = reinterpret_cast<float*>(sh_lane_raw);
  char* s_mem = reinterpret_cast<char*>(s_boys + SH_BOYS_K * SH_BOYS_ROW);
  __shared__ double s_red[4][64];
  const int cta = A.cta0 + (int)blockIdx.x;
  const ShWork W = A.work[A.lcta[cta]];
  const int unit = cta - W.lcta0;  // [component chunk][bra block][ket chunk]
  const int ch = unit / W.lsplit, r = unit - ch * W.lsplit;
  const int blk = r / W.nkc, kc = r - blk * W.nkc;
  if (A.pair[W.bra].d != DB || A.pair[W.ket].nterm != KET::S.nterm || A.pair[W.bra].ncomp * NF > 64) return;
  lane_chunk<KET, DB, 0, NF, ONE4>(ch, A, W, blk, kc, s_boys, s_mem, s_red);
}

template <int TA, int TB, bool SAME, bool OC, int DB, bool ONE4>
cudaError_t launch_lane(int ncta, cudaStream_t st, const ShArgs& A) {
  using KET = LaneKet<TA, TB, SAME, OC>;
  constexpr int NF = sh_lane_chunk(DB, TA, TB), H = sh_nherm(DB);
  constexpr size_t sums = 4 * sizeof(df) * H * NF * 33, ket = LaneDim<KET, DB>::ket_bytes;
  constexpr size_t smem = sizeof(float) * SH_BOYS_K * SH_BOYS_ROW + (sums > ket ? sums : ket);
  static_assert(smem <= 100 * 1024, "two CTAs per SM");
  auto kern = shell_lane_kernel<KET, DB, NF, ONE4>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<ncta, SH_LANE_BRA, smem, st>>>(A);
  return cudaGetLastError();
}

// dispatch of one ket type over the bra degrees that have a kernel
template <int TA, int TB, bool SAME, bool OC, bool ONE4, int DB = 0>
cudaError_t launch_lane_bra(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  if constexpr (DB > 4) {
    return cudaErrorInvalidValue;
  } else {
    if constexpr (sh_lane_chunk(DB, TA, TB) > 0)
      if (db == DB) return launch_lane<TA, TB, SAME, OC, DB, ONE4>(ncta, st, A);
    return launch_lane_bra<TA, TB, SAME, OC, ONE4, DB + 1>(db, ncta, st, A);
  }
}

#endif  // __CUDACC__

}  // namespace ss
