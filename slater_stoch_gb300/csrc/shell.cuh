// shell.cuh -- data of the shell-quartet ERI path: shells, shell pairs, their primitive records
// and Hermite expansions.
//
// A shell is the set of functions that share centre and Gaussian fit: s, p, the six cartesian d's,
// or one r^2-type fit ("r", a d shell contracted to x^2 + y^2 + z^2).  All its components share
// the primitive exponents and coefficients, so everything of a primitive quartet that depends
// only on exponents and centres -- the Gaussian products, the Boys function and the Hermite
// integrals -- is formed once per primitive quartet of four shells instead of once per function
// quartet (the reference's gauss_ijkl, src/gauss_ijkl.F90:51-154, works function by function).
#pragma once
#include <stdint.h>

#include "ss_common.cuh"

namespace ss {

// Shell types in the canonical order of a pair (the larger type first).
enum { SH_S = 0, SH_P = 1, SH_R = 2, SH_D = 3 };
constexpr int SH_NBASE = 10;                 // SS PS PP RS RP RR DS DP DR DD
constexpr int SH_NSTRUCT = 2 * (SH_NBASE + 2);  // + one shell with itself (PP, DD); x one centre
constexpr int SH_MAXCOMP = 36;
constexpr int SH_MAXTERM = 342;              // DD on two centres
constexpr int SH_MAXL = 8;
constexpr int SH_MAXH = 35;                  // Hermite functions of degree <= 4

// Hermite functions of total degree n = t + u + v, ordered by degree
__host__ __device__ constexpr int sh_nherm(int d) { return (d + 1) * (d + 2) * (d + 3) / 6; }
__host__ __device__ constexpr int sh_hidx(int t, int u, int v) {
  return (t + u + v) * (t + u + v + 1) * (t + u + v + 2) / 6 + (u + v) * (u + v + 1) / 2 + v;
}
// packed degrees x | y << 8 | z << 16
__host__ __device__ constexpr int sh_pack_idx(uint32_t h) {
  return sh_hidx((int)(h & 255), (int)((h >> 8) & 255), (int)(h >> 16));
}

// Sparsity of a pair type: which Hermite functions each component's charge distribution has.
struct ShStruct {
  int d, ncomp, nterm, pad;          // degree, components, total number of terms
  int fs[SH_MAXCOMP + 1];            // first term of each component
  uint32_t term[SH_MAXTERM];         // packed degrees
  int ncombo[SH_MAXCOMP];            // cartesian products whose sum is the component (r: x^2 + y^2 + z^2)
  uint32_t combo[SH_MAXCOMP][9];     // packed powers of the two functions: 4 bits each ax ay az bx by bz
};

constexpr int SH_DEG[4] = {0, 1, 2, 2};  // S P R D
constexpr int SH_NC[4] = {1, 3, 1, 6};
constexpr int SH_POW[4][6][3] = {{{0, 0, 0}},
                                 {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}},
                                 {{0, 0, 0}},
                                 {{2, 0, 0}, {1, 1, 0}, {1, 0, 1}, {0, 2, 0}, {0, 1, 1}, {0, 0, 2}}};

// Pair type of canonical shell types ta >= tb; same: one shell with itself (components ca >= cb);
// onec: both shells on one centre.  Components ca-major; a component's terms in (t, u, v) order.
constexpr ShStruct sh_struct(int ta, int tb, bool same, bool onec) {
  ShStruct S{};
  S.d = SH_DEG[ta] + SH_DEG[tb];
  int nterm = 0;
  for (int ca = 0; ca < SH_NC[ta]; ca++)
    for (int cb = 0; cb < SH_NC[tb]; cb++) {
      if (same && cb > ca) continue;
      const int f = S.ncomp++;
      const int na = ta == SH_R ? 3 : 1, nb = tb == SH_R ? 3 : 1;
      int pa[9][3] = {}, pb[9][3] = {};
      for (int x = 0; x < na; x++)
        for (int y = 0; y < nb; y++) {
          const int k = S.ncombo[f]++;
          uint32_t code = 0;
          for (int ax = 0; ax < 3; ax++) {
            pa[k][ax] = ta == SH_R ? (ax == x ? 2 : 0) : SH_POW[ta][ca][ax];
            pb[k][ax] = tb == SH_R ? (ax == y ? 2 : 0) : SH_POW[tb][cb][ax];
            code |= (uint32_t)pa[k][ax] << (4 * ax) | (uint32_t)pb[k][ax] << (4 * (3 + ax));
          }
          S.combo[f][k] = code;
        }
      S.fs[f] = nterm;
      for (int t = 0; t <= S.d; t++)
        for (int u = 0; t + u <= S.d; u++)
          for (int v = 0; t + u + v <= S.d; v++) {
            const int h[3] = {t, u, v};
            bool any = false;
            for (int k = 0; k < S.ncombo[f]; k++) {
              bool ok = true;
              for (int ax = 0; ax < 3; ax++) {
                const int e = pa[k][ax] + pb[k][ax];
                ok = ok && h[ax] <= e && !(onec && ((e - h[ax]) & 1));  // on one centre only equal parities
              }
              any = any || ok;
            }
            if (any) S.term[nterm++] = (uint32_t)(t | (u << 8) | (v << 16));
          }
    }
  S.fs[S.ncomp] = nterm;
  S.nterm = nterm;
  return S;
}

// One shell pair of a system.  Its primitives occupy prim[prim_off .. prim_off + cap), cnt[pair] of them used.
struct ShPair {
  int st, d, ncomp, nterm;
  int cap;                           // most primitives it can have after the K_AB screen
  int fa, fb;                        // one function of each shell (exponents, coefficients, centre)
  int onec, fold;
  int64_t prim_off, e_off;           // first primitive; first Hermite coefficient
  int col[5];                        // where ShArgs::col has this pair type's columns as the ket, by bra degree
};

// A primitive pair: exponent sum, centre, w = K_AB c_a c_b / p, and (sorted tables) the largest
// Schwarz factor of its components relative to the function pairs' own diagonals.
struct ShPrim {
  double p, P[3], w, S;
};
// Two-float view (high and low parts); w is divided by the pair's power of two (ShArgs::scale).  The
// centre has a third part, so that the distance of two centres keeps two-float accuracy wherever the
// molecule lies.  s is the power of two next below sqrt(2 p), is = 1 / s: the primitive's unit of
// length in the FP32 evaluations (shell_eri.cuh).
struct ShPrimF {
  float p[2], ph[3], pl[3], pm[3], w[2], s, is, pad;
};
static_assert(sizeof(ShPrimF) % sizeof(float4) == 0, "the records are copied as float4");

// One shell quartet of a launch.
struct ShWork {
  int bra, ket;          // shell pairs
  int cta0, split;       // first CTA, number of bra slices
  int lane, lcta0, nlane;  // lane kernel: instance (-1: none), first CTA, CTAs
  int lsplit, nkc;       // its partial sums per element (bra blocks x ket chunks), ket chunks
  int64_t part, elem;    // first partial sum [element][split + lsplit]; first element of the result
  uint64_t mask;         // ket components that are asked for
};

// Boys tables of one top degree L, row k around T_k = k/8, a_j = F_{L+j}(T_k) / j!: FP64 a_0..a_8,
// and for the FP32 evaluations a_0..a_4 and e^-T_k as two floats and a_5..a_8 (rows of 20 floats:
// 16-byte loads of different rows spread over the banks).
constexpr int SH_BOYS_K = 289, SH_BOYS_ROW = 20;
struct alignas(16) ShBoys {
  float f[SH_BOYS_K][SH_BOYS_ROW];
  double a[SH_BOYS_K][9];
};
static_assert(sizeof(ShBoys) % 16 == 0 && sizeof(float) * SH_BOYS_K * SH_BOYS_ROW % 16 == 0 && SH_BOYS_ROW % 4 == 0,
              "the FP32 tables are copied and read as float4");

struct ShArgs {
  const ShPair* pair;
  const int* cnt;
  const ShPrim* prim;
  const ShPrimF* primf;
  const double* E;
  const float2* E2;      // E_t s^|t| as two floats, s of the primitive
  const double* scale;   // power of two of each pair's w in primf
  const ShBoys* boys;    // [SH_MAXL + 1]
  const uint8_t* col;    // columns of t + tau of every bra degree and pair type (ShPair::col)
  const ShStruct* st;
  const ShWork* work;
  const int* cta;        // work entry of each CTA of the chunk
  int cta0;              // first CTA of this launch in it
  double* partial;
  const int* lcta;       // the same for the lane kernels
  double eps, eps32, eps_df;
  int diag;              // 1: (P|Q) of a pair with itself, Q <= P, diagonal elements only
};

constexpr int SH_SMEM_MAX = 200 * 1024;
constexpr int SH_MAXSLICE = 16;  // bra primitives of a slice

cudaError_t launch_shell_eri(int L, int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A);

// Bytes of the columns [ket term][bra Hermite function] of a bra degree and a pair type: indices of
// t + tau, in multiples of 16 bytes
__host__ __device__ constexpr int sh_col_size(int d, int nterm) { return (sh_nherm(d) * nterm + 15) / 16 * 16; }

// Lane kernels (shell_lane.cuh): bra degree DB, ket type; a CTA takes SH_LANE_BRA bra primitives (one
// per thread), sh_lane_kets ket primitives and one chunk of the ket's components.  Fewer kets where a
// ket costs more: on a small system the longest CTA is the stage, and its start-up (the Boys table)
// is about one ket's work there (7-function water 1.64 ms with 64 kets at every L, 1.40 ms with 32
// from L = 3; 26-function water 44.3 ms with both).
constexpr int SH_LANE_BRA = 128;
constexpr int sh_lane_kets(int L) { return L >= 3 ? 32 : 64; }
// ket components per chunk for a bra of degree db and a ket type (ta, tb), 0: no such kernel
constexpr int sh_lane_chunk(int db, int ta, int tb) {
  const int k = ta * (ta + 1) / 2 + tb;  // SS PS PP RS RP RR DS DP DR DD
  if (k == 0) return db <= 4 ? 1 : 0;                                        // SS
  if (k == 1) return db == 1 || db == 2 ? 3 : (db == 3 || db == 4 ? 1 : 0);  // PS
  if (k == 2) return db == 2 ? 3 : 0;                                        // PP
  if (k == 3) return db >= 1 && db <= 3 ? 1 : 0;                             // RS
  if (k == 4) return db == 1 || db == 2 ? 3 : (db == 3 ? 1 : 0);             // RP
  if (k == 5) return db == 1 || db == 2 ? 1 : 0;                             // RR
  if (k == 6) return db == 2 ? 3 : 0;                                        // DS
  if (k == 8) return db == 1 ? 3 : 0;                                        // DR
  return 0;
}
// instance = 8 * (pair type index) + bra degree, + SH_LANE_ONEC where all four shells are on one centre
constexpr int SH_LANE_ONEC = 1024;
cudaError_t launch_shell_lane(int instance, int ncta, cudaStream_t st, const ShArgs& A);

}  // namespace ss
