// shell_basis.h -- shells of a fitted basis and their pairs (host code, no CUDA calls).
#pragma once
#include <stdint.h>

#include <utility>
#include <vector>

#include "shell.cuh"

namespace ss {

// pair type of canonical shell types ta >= tb; same: one shell with itself (components ca >= cb)
inline int struct_index(int ta, int tb, bool same, bool onec) {
  int base = ta * (ta + 1) / 2 + tb;
  if (same && ta == SH_P) base = SH_NBASE;
  if (same && ta == SH_D) base = SH_NBASE + 1;
  return 2 * base + (onec ? 1 : 0);
}

struct StructTable {
  std::vector<ShStruct> s;
  std::vector<uint8_t> col;         // ShArgs::col
  int off[SH_NSTRUCT][5] = {};
  StructTable() : s(SH_NSTRUCT) {
    for (int ta = 0; ta < 4; ta++)
      for (int tb = 0; tb <= ta; tb++)
        for (int oc = 0; oc < 2; oc++) s[struct_index(ta, tb, false, oc)] = sh_struct(ta, tb, false, oc);
    for (int oc = 0; oc < 2; oc++) {
      s[struct_index(SH_P, SH_P, true, oc)] = sh_struct(SH_P, SH_P, true, oc);
      s[struct_index(SH_D, SH_D, true, oc)] = sh_struct(SH_D, SH_D, true, oc);
    }
    for (int st = 0; st < SH_NSTRUCT; st++)
      for (int d = 0; d < 5; d++) {
        const ShStruct& S = s[st];
        off[st][d] = (int)col.size();
        col.resize(col.size() + sh_col_size(d, S.nterm));
        for (int x = 0; x < S.nterm; x++)
          for (int n = 0, t = 0; n <= d; n++)  // bra Hermite functions in the order of sh_hidx
            for (int w = 0; w <= n; w++)
              for (int v = 0; v <= w; v++, t++) {
                const uint32_t tm = S.term[x];
                col[off[st][d] + x * sh_nherm(d) + t] = (uint8_t)sh_hidx(
                    n - w + (int)(tm & 255), w - v + (int)((tm >> 8) & 255), v + (int)(tm >> 16));
              }
      }
  }
};
inline const StructTable& structs() {
  static const StructTable t;
  return t;
}

// Host view of a fitted basis (the layouts of BasisDev); sys: system of each function, in
// non-decreasing order, or null for one system.
struct BasisHost {
  int n, ld;
  const double* center;
  const int *npower, *i_type, *n_gauss;
  const double *c_gauss, *g_gauss;
  const int* sys;
};

// Shells of the basis and the pairs of every two shells of one system.  Pairs across systems do not
// exist: the tables of a batch grow with its systems, not with their square.
struct ShellBasis {
  bool all = true;                   // every function is in a shell
  std::vector<int> fsh, fcomp;       // shell (-1: in none) and component of every function
  std::vector<int> sys, nb;          // system and number of components of every shell
  std::vector<int> first;            // first shell of every system, and the end
  std::vector<int64_t> at;           // where a system's nsh x nsh block of spair and flip begins
  std::vector<int> spair;            // pair of every two shells of a system
  std::vector<char> flip;            // whether the pair holds them in the other order
  std::vector<int> pfirst;           // first pair of every system, and the end
  std::vector<ShPair> pair;
  int64_t nprim = 0, nE = 0;

  // shell pair and component of functions i and k; false if one is in no shell, or across systems
  bool component(int i, int k, int* pr, int* comp) const {
    int a = fsh[i], b = fsh[k];
    if (a < 0 || b < 0 || sys[a] != sys[b]) return false;
    const int s = sys[a], ns = first[s + 1] - first[s];
    const int64_t o = at[s];
    int ca = fcomp[i], cb = fcomp[k];
    if (flip[o + (int64_t)(a - first[s]) * ns + (b - first[s])]) {
      std::swap(a, b);
      std::swap(ca, cb);
    }
    *pr = spair[o + (int64_t)(a - first[s]) * ns + (b - first[s])];
    if (a == b) {
      if (ca < cb) std::swap(ca, cb);
      *comp = ca * (ca + 1) / 2 + cb;
    } else {
      *comp = ca * nb[b] + cb;
    }
    return true;
  }
};

// A function beyond d, or an r^2-type fit with angular factors, belongs to no shell: its quartets
// take the per-function kernel (eri_kernel.cuh).
inline ShellBasis build_shell_basis(const BasisHost& B) {
  ShellBasis T;
  const int n = B.n, ld = B.ld;
  T.fsh.assign(n, -1);
  T.fcomp.assign(n, 0);
  std::vector<int> rep, type;  // one function and the type of every shell
  auto same_fit = [&](int a, int b) {
    if (B.n_gauss[a] != B.n_gauss[b] || B.i_type[a] != B.i_type[b]) return false;
    const size_t t = B.i_type[a] == 2 ? 1 : 0;
    for (int m = 0; m < B.n_gauss[a]; m++)
      if (B.g_gauss[m + (size_t)ld * a] != B.g_gauss[m + (size_t)ld * b] ||
          B.c_gauss[m + (size_t)ld * (a + n * t)] != B.c_gauss[m + (size_t)ld * (b + n * t)])
        return false;
    return true;
  };
  auto same_centre = [&](int a, int b) {
    for (int ax = 0; ax < 3; ax++)
      if (B.center[3 * a + ax] != B.center[3 * b + ax]) return false;
    return true;
  };
  // At least as many as the primitives that shell_fill keeps: its cuts are exponents
  // a b r2 / (a + b) above 40 and factors below 1e-15, whose exponent is 34.5388; 34.6 leaves room
  // for the rounding of both sides.
  auto kept = [&](int f, int g) {
    double r2 = 0.0;
    for (int ax = 0; ax < 3; ax++) {
      const double x = B.center[3 * f + ax] - B.center[3 * g + ax];
      r2 += x * x;
    }
    int count = 0;
    for (int m = 0; m < B.n_gauss[f]; m++) {
      const double a = B.g_gauss[m + (size_t)ld * f];
      for (int k = 0; k < B.n_gauss[g]; k++) {
        const double b = B.g_gauss[k + (size_t)ld * g];
        count += !(a * b * r2 > 34.6 * (a + b));
      }
    }
    return count;
  };
  int64_t po = 0, eo = 0;
  T.first.push_back(0);
  T.pfirst.push_back(0);
  for (int f0 = 0, f1 = 0; f0 < n; f0 = f1) {
    for (f1 = f0 + 1; f1 < n && !(B.sys && B.sys[f1] != B.sys[f0]);) f1++;
    const int s0 = (int)rep.size();
    for (int f = f0; f < f1; f++) {
      const int* np = &B.npower[3 * f];
      const int l = np[0] + np[1] + np[2];
      if (B.i_type[f] == 2 ? l > 0 : l > 2) {
        T.all = false;
        continue;
      }
      const int ty = B.i_type[f] == 2 ? SH_R : (l == 0 ? SH_S : l == 1 ? SH_P : SH_D);
      int comp = 0;
      for (int x = 0; x < SH_NC[ty]; x++)
        if (ty != SH_R && SH_POW[ty][x][0] == np[0] && SH_POW[ty][x][1] == np[1] && SH_POW[ty][x][2] == np[2]) comp = x;
      T.fcomp[f] = comp;
      // a shell with this fit (components are mostly consecutive: the latest shells first)
      for (int s = (int)rep.size() - 1; s >= s0 && T.fsh[f] < 0; s--)
        if (type[s] == ty && same_centre(rep[s], f) && same_fit(rep[s], f)) T.fsh[f] = s;
      if (T.fsh[f] < 0) {
        T.fsh[f] = (int)rep.size();
        rep.push_back(f);
        type.push_back(ty);
        T.sys.push_back((int)T.first.size() - 1);
        T.nb.push_back(SH_NC[ty]);
      }
    }
    const int ns = (int)rep.size() - s0;
    const int64_t o = (int64_t)T.spair.size();
    T.at.push_back(o);
    T.spair.resize(o + (int64_t)ns * ns, -1);
    T.flip.resize(o + (int64_t)ns * ns, 0);
    for (int x = 0; x < ns; x++)
      for (int y = 0; y <= x; y++) {
        int a = x, b = y;
        if (type[s0 + a] < type[s0 + b]) std::swap(a, b);
        ShPair P{};
        P.fa = rep[s0 + a];
        P.fb = rep[s0 + b];
        P.onec = same_centre(P.fa, P.fb);
        P.fold = P.onec && same_fit(P.fa, P.fb);
        P.st = struct_index(type[s0 + a], type[s0 + b], a == b, P.onec);
        const ShStruct& S = structs().s[P.st];
        P.d = S.d;
        P.ncomp = S.ncomp;
        P.nterm = S.nterm;
        for (int d = 0; d < 5; d++) P.col[d] = structs().off[P.st][d];
        const int na = B.n_gauss[P.fa], nb = B.n_gauss[P.fb];
        P.cap = P.fold ? na * (na + 1) / 2 : P.onec ? na * nb : kept(P.fa, P.fb);
        P.prim_off = po;
        P.e_off = eo;
        po += P.cap;
        eo += (int64_t)P.cap * P.nterm;
        // (x, y) as given is (b, a) of the pair
        T.spair[o + (int64_t)x * ns + y] = T.spair[o + (int64_t)y * ns + x] = (int)T.pair.size();
        T.flip[o + (int64_t)b * ns + a] = a != b;
        T.pair.push_back(P);
      }
    T.first.push_back((int)rep.size());
    T.pfirst.push_back((int)T.pair.size());
  }
  T.nprim = po;
  T.nE = eo;
  return T;
}

}  // namespace ss
