// mc.cuh -- device views and launchers of the ZV-MC kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ss_common.cuh"

namespace ss {

// Used pairs (i,k), i >= k, in groups with the same ZV map and radial parts: all components of two
// shells (src/two_e_slater.F90:339-348,406).  Group g: functions i[g], k[g] (any of its pairs),
// pairs order[first[g]] .. order[first[g + 1] - 1].
struct ZvPairs {
  int ngroups;
  const int* i;
  const int* k;
  const int* same;     // both functions have the same centre and radial part
  const int* first;
  const int* order;
  const int* pi;       // functions of each pair
  const int* pk;
  const double* G;     // [3*ngroups] centre of the map
  const double* fzv;   // 0.5 a_ZV / (zeta_i + zeta_k)
  const double* fjac;  // a_ZV / (zeta_i + zeta_k)
};

// per-chunk columns, [group or pair][walker] with leading dimension ld (walker fastest)
struct ZvChunk {
  int64_t ld;
  double *u1x, *u1y, *u1z, *u2x, *u2y, *u2z;  // per group
  double *a_s, *a_g, *b_s, *b_g;  // per pair; FP64: J1 rhoS1, J1 rhoG1, J2 rhoS2/pi0, J2 rhoG2/pi0; REF32: raw densities
  double *j1, *j2;                // per group, REF32 only
};

// Up to ZV_TB x ZV_TK quartets whose bra pairs are in one group and whose ket pairs are in one group.
// Bit t * ZV_TK + u of mask: the quartet (bra[t] | ket[u]), whose index is the next of ZvTiles::q from
// q.  6 x 6: the most whose sums (144 registers) stay in registers.
constexpr int ZV_TB = 6, ZV_TK = 6;
struct ZvTile {
  uint64_t mask;
  int64_t q;
  int g1, g2;
  int bra[ZV_TB], ket[ZV_TK];  // -1: no quartet has it
};
struct ZvTiles {
  int n;
  const ZvTile* tile;
  const int64_t* q;
};

cudaError_t launch_draw_walkers(cudaStream_t st, uint64_t seed, int64_t first, int64_t S, double* r1,
                                double* r2);
cudaError_t launch_walker_aux(cudaStream_t st, int64_t S, const double* r1, const double* r2, double* r1m,
                              double* r2m, double* pi0);
cudaError_t launch_zv_pairs(cudaStream_t st, int mode, const BasisDev& B, const ZvPairs& P,
                            int64_t S, const double* r1, const double* r2, const double* r1m,
                            const double* r2m, const double* pi0, const ZvChunk& Z);
cudaError_t launch_zv_accum(cudaStream_t st, int mode, int nsplit, int64_t S, const ZvTiles& Q,
                            const ZvChunk& Z, const double* pi0, double* partS, double* partG);
cudaError_t launch_zv_reduce(cudaStream_t st, int64_t nint, int nsplit, const double* partS,
                             const double* partG, double* eS, double* eG);
cudaError_t launch_zv_block_stats(cudaStream_t st, int64_t nint, int64_t npts, double* eS, double* eG,
                                  double* acc, double* acc2);
cudaError_t launch_zv_final(cudaStream_t st, int64_t nint, int nb, int unbiased, const double* acc,
                            const double* acc2, double* mean, double* sigma, unsigned long long* maxbits);

}  // namespace ss
