// Host build of the two-float arithmetic (csrc/df32.cuh) and of the shell-quartet kernels' Boys
// functions (csrc/shell_eri.cuh), for test_df32_host.py.  IEEE arithmetic with explicit fma: the
// device's, except for the reciprocal square roots' seeds and expf, which CUDA rounds its own way.
#include <cmath>
#include <memory>

#include "../slater_stoch_gb300/csrc/boys_grid.cuh"
#include "../slater_stoch_gb300/csrc/shell_eri.cuh"

using namespace ss;

static df get(const float* a) { return df{a[0], a[1]}; }
static void put(float* o, df v) {
  o[0] = v.h;
  o[1] = v.l;
}

// op 0: a + b, 1: a * b, 2: a * b + c, 3: 1/sqrt(a), 4: difference of three floats (a: 3, b: 3)
extern "C" void ss_host_df(int op, int n, const float* a, const float* b, const float* c, float* out) {
  for (int i = 0; i < n; i++) {
    df v{0.f, 0.f};
    if (op == 0) v = df_add(get(a + 2 * i), get(b + 2 * i));
    if (op == 1) v = df_mul(get(a + 2 * i), get(b + 2 * i));
    if (op == 2) v = df_fma(get(a + 2 * i), get(b + 2 * i), get(c + 2 * i));
    if (op == 3) v = df_rsqrt(get(a + 2 * i));
    if (op == 4) v = df_sub3(a[3 * i], a[3 * i + 1], a[3 * i + 2], b[3 * i], b[3 * i + 1], b[3 * i + 2]);
    put(out + 2 * i, v);
  }
}

// the tables of one top degree, as shell_boys (csrc/shell_tables.cu) fills them
static void fill(ShBoys* out, int L) {
  for (int k = 0; k < SH_BOYS_K; k++) {
    double fact = 1.0;
    float* f = out->f[k];
    for (int j = 0; j < 9; j++) {
      if (j > 1) fact *= j;
      const double a = boys_grid_tab[k * BOYS_GRID_N + L + j] / fact;
      out->a[k][j] = a;
      if (j < 5) {
        f[2 * j] = (float)a;
        f[2 * j + 1] = (float)(a - (double)(float)a);
      } else {
        f[12 + j - 5] = (float)a;
      }
    }
    const double e = std::exp(-0.125 * k);
    f[10] = (float)e;
    f[11] = (float)(e - (double)(float)e);
  }
}

template <int L>
static void boys_all(const ShBoys* tab, int n, const double* T, double* f64, double* f48, double* f32) {
  for (int i = 0; i < n; i++) {
    double F[L + 1];
    df G[L + 1];
    float H[L + 1];
    boys_shell<L>(T[i], F, tab);
    boys_shell<L>(df_from(T[i]), G, &tab->f[0][0]);
    boys_shell<L>((float)T[i], H, &tab->f[0][0]);
    for (int m = 0; m <= L; m++) {
      f64[9 * i + m] = F[m];
      f48[9 * i + m] = df_to(G[m]);
      f32[9 * i + m] = (double)H[m];
    }
  }
}

// out[9 i + m] = F_m(T[i]), m = 0..L, in the three types
extern "C" int ss_host_shell_boys(int L, int n, const double* T, double* f64, double* f48, double* f32) {
  auto tab = std::make_unique<ShBoys>();
  fill(tab.get(), L);
  switch (L) {
    case 0: boys_all<0>(tab.get(), n, T, f64, f48, f32); return 0;
    case 1: boys_all<1>(tab.get(), n, T, f64, f48, f32); return 0;
    case 4: boys_all<4>(tab.get(), n, T, f64, f48, f32); return 0;
    case 8: boys_all<8>(tab.get(), n, T, f64, f48, f32); return 0;
  }
  return -1;
}
