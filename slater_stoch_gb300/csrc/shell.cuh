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

// One shell pair.  Its primitives occupy prim[prim_off .. prim_off + cap), cnt[pair] of them used.
struct ShPair {
  int st, d, ncomp, nterm;
  int cap;                           // most primitives it can have (before the K_AB screen)
  int fa, fb;                        // one function of each shell (exponents, coefficients, centre)
  int onec, fold, same_system;
  int64_t prim_off, e_off;           // first primitive; first Hermite coefficient
  double pmax;                       // largest exponent sum of its primitives
};

// A primitive pair: exponent sum, centre, w = K_AB c_a c_b / p, and (sorted tables) the largest
// Schwarz factor of its components relative to the function pairs' own diagonals.
struct ShPrim {
  double p, P[3], w, S;
};
// Two-float view (high and low parts); w is divided by the pair's power of two (ShArgs::scale)
struct ShPrimF {
  float p[2], ph[3], pl[3], w[2], pad[2];
};
static_assert(sizeof(ShPrim) == 48 && sizeof(ShPrimF) == 48, "primitive records are 48 bytes");

// One shell quartet of a launch.
struct ShWork {
  int bra, ket;          // shell pairs
  int cta0, split;       // first CTA, number of bra slices
  int64_t part, elem;    // first partial sum [element][slice]; first element of the result
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
  const float2* E2;      // the same as two floats
  const double* scale;   // power of two of each pair's w in primf
  const ShBoys* boys;    // [SH_MAXL + 1]
  const ShStruct* st;
  const ShWork* work;
  const int* cta;        // work entry of each CTA of the chunk
  int cta0;              // first CTA of this launch in it
  double* partial;
  double eps, eps32, eps_df;
  int diag;              // 1: (P|Q) of a pair with itself, Q <= P, diagonal elements only
};

constexpr int SH_SMEM_MAX = 200 * 1024;

cudaError_t launch_shell_eri(int L, int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A);

}  // namespace ss
