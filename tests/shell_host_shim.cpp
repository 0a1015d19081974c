// Host build of the shell tables' sizes (slater_stoch_gb300/csrc/shell_basis.h).
#include "../slater_stoch_gb300/csrc/shell_basis.h"

using namespace ss;

// out: shells, pairs, primitives, Hermite coefficients; cap[pair], fa[pair], fb[pair] up to max_pair;
// fn_pair[i * n + k] (i >= k): the pair of functions i and k, -1 if there is none
extern "C" int ss_host_shells(int n, int ld, const double* center, const int* npower, const int* i_type, const int* n_gauss,
                              const double* c_gauss, const double* g_gauss, const int* sys, int64_t* out, int max_pair,
                              int* cap, int* fa, int* fb, int* fn_pair) {
  const ShellBasis T = build_shell_basis(BasisHost{n, ld, center, npower, i_type, n_gauss, c_gauss, g_gauss, sys});
  out[0] = (int64_t)T.nb.size();
  out[1] = (int64_t)T.pair.size();
  out[2] = T.nprim;
  out[3] = T.nE;
  if ((int)T.pair.size() > max_pair) return -1;
  for (size_t x = 0; x < T.pair.size(); x++) {
    cap[x] = T.pair[x].cap;
    fa[x] = T.pair[x].fa;
    fb[x] = T.pair[x].fb;
  }
  for (int i = 0; i < n; i++)
    for (int k = 0; k <= i; k++) {
      int p = -1, f = 0;
      fn_pair[(int64_t)i * n + k] = T.component(i, k, &p, &f) ? p : -1;
    }
  return 0;
}
