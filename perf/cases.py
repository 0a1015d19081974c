"""The workloads by which this framework's speed is judged: what they are, how their inputs are
made, one pass of each through the public entry points, the work a pass cannot do without, and
(where it can be had in a few seconds) its result in plain 64-bit torch.

Systems.  ``water7`` and ``water26`` are the H2O bases of ``slater_stoch_gb300/configs.py``;
``mol`` is a molecule by the rules of its ``random_molecule`` (H 1s 2p, heavy atoms 1s 2s 2p 3d,
Slater-rule exponents) with the listed atoms.  The seed moves the nuclei and the exponents, so
every seed is another input of the same shape.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from slater_stoch_gb300 import api, basis, batch, configs

A_ZV = 1.8
HEAVY = ("1S", "2S", "2P", "3D")
LIGHT = ("1S", "2P")


# ---- the cases -------------------------------------------------------------------------------
def listed():
    return [
        # analytic ERIs of the fits, the stage every job starts with: a minimal basis (the smallest
        # call, bound by launches and host work), ...
        {"name": "eri_water7", "kind": "eri", "system": "water7", "ng0": 20},
        # ... one heavy atom (a serving request: every integral on one centre), ...
        {"name": "eri_atom", "kind": "eri", "system": "mol", "atoms": "O", "ng0": 20},
        # ... a diatomic with fits of an odd length, ...
        {"name": "eri_diatomic", "kind": "eri", "system": "mol", "atoms": "C O", "ng0": 17},
        # ... and the 26-function water of the benchmark
        {"name": "eri_water26", "kind": "eri", "system": "water26", "ng0": 20},
        # the whole two-electron job: the benchmark's (2^26 walker pairs), ...
        {"name": "job_water26", "kind": "job", "system": "water26", "ng0": 20, "npts": 1 << 22, "nblocks": 16},
        # ... and one serving request (one atom, two blocks of 2^16 walker pairs)
        {"name": "job_atom", "kind": "job", "system": "mol", "atoms": "N", "ng0": 20, "npts": 1 << 16, "nblocks": 2},
        # many small systems of uneven size in one call (the batched workload)
        {"name": "batch_small", "kind": "batch", "systems": "O|H H|N|H|O H|C|H", "ng0": 20, "npts": 1 << 16, "nblocks": 2},
        # more Monte Carlo on a resident system: the shared walkers on the tensor cores, ...
        {"name": "mc_shared", "kind": "mc", "system": "water26", "ng0": 20, "npts": 1 << 20, "nblocks": 4,
         "estimator": "shared", "precision": "split_bf16"},
        # ... and the reference's own per-pair estimator in FP64
        {"name": "mc_faithful", "kind": "mc", "system": "water26", "ng0": 20, "npts": 4000, "nblocks": 4,
         "estimator": "faithful", "precision": "fp64"},
        # cleanup of the noisy ERI matrix: randomized SVD deflation with the benchmark's parameters, ...
        {"name": "clean_svd", "kind": "svd", "n": 26, "layout": "packed_pair", "rank": 200, "oversample": 10, "q": 4},
        # ... and the exact projection
        {"name": "clean_project", "kind": "project", "n": 26, "layout": "packed_pair"},
        # one-electron integrals of a new system
        {"name": "one_e_water26", "kind": "one_e", "system": "water26", "ng0": 20},
    ]


_ATOMS = ["H", "O", "H H", "C H", "N H", "O H H", "C N", "O C", "C O H"]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def system(small):
        if rng.random() < 0.25:
            return {"system": "water7", "ng0": rng.randint(9, 20)}
        atoms = rng.choice(_ATOMS[:6] if small else _ATOMS)
        return {"system": "mol", "atoms": atoms, "ng0": rng.randint(10, 20 if len(atoms) < 5 else 18)}

    kind = rng.choice(["eri", "eri", "job", "mc", "mc", "batch", "svd", "project", "one_e"])
    if kind == "eri":
        return {"kind": "eri", **system(False)}
    if kind == "job":
        return {"kind": "job", **system(True), "npts": logint(1 << 13, 1 << 20), "nblocks": rng.randint(2, 4)}
    if kind == "mc":
        if rng.random() < 0.5:
            return {"kind": "mc", **system(False), "npts": logint(1 << 13, 1 << 21), "nblocks": rng.randint(2, 4),
                    "estimator": "shared", "precision": "split_bf16"}
        return {"kind": "mc", **system(False), "npts": 40 * logint(10, 300), "nblocks": rng.randint(2, 4),
                "estimator": "faithful", "precision": rng.choice(["fp64", "ref32"])}
    if kind == "batch":
        return {"kind": "batch", "systems": "|".join(rng.choice(_ATOMS[:5]) for _ in range(rng.randint(2, 8))),
                "ng0": rng.randint(10, 20), "npts": logint(1 << 13, 1 << 17), "nblocks": rng.randint(2, 3)}
    n = rng.randint(7, 28)
    if kind == "svd":
        N = n * (n + 1) // 2
        return {"kind": "svd", "n": n, "layout": "packed_pair", "rank": rng.randint(N // 3, (2 * N) // 3),
                "oversample": rng.randint(0, 12), "q": rng.randint(2, 4)}
    if kind == "project":
        return {"kind": "project", "n": n, "layout": "packed_pair"}
    return {"kind": "one_e", **system(False)}


# ---- inputs ----------------------------------------------------------------------------------
def _molecule(symbols, coords, per_element, ng0):
    mol = basis.molecule_bohr(symbols, coords)
    return mol, basis.build_basis(mol, per_element, basis.FitParams(ng0=ng0))


def _mol(atoms, ng0, rng):
    syms = atoms.split()
    side = 2.0 + 2.0 * len(syms) ** (1.0 / 3.0)
    pos = []
    while len(pos) < len(syms):
        p = rng.uniform(0.0, side, size=3)
        if all(np.linalg.norm(p - q) >= 2.0 for q in pos):
            pos.append(p)
    per = {}
    for s in syms:
        z = basis.element_number(s)
        per[z] = [(o, configs.SLATER[z][o] * rng.uniform(0.8, 1.2)) for o in (LIGHT if z == 1 else HEAVY)]
    return _molecule(syms, np.array(pos), per, ng0)


def _system(case, seed):
    rng = np.random.default_rng(1000003 * seed + 17)
    if case["system"] == "mol":
        return _mol(case["atoms"], case["ng0"], rng)
    if case["system"] == "water7":
        per = {8: [("1S", 7.66), ("2S", 2.25), ("2P", 2.25)], 1: [("1S", 1.24)]}
    else:
        per = {8: [("1S", 7.9), ("1S", 6.6), ("2S", 2.7), ("2S", 1.7), ("2P", 2.9), ("2P", 1.5), ("3D", 2.0)],
               1: [("1S", 1.6), ("1S", 1.0), ("2P", 1.3)]}
    per = {z: [(o, x * rng.uniform(0.97, 1.03)) for o, x in v] for z, v in per.items()}
    xyz = np.array(configs.H2O_BOHR) + rng.uniform(-0.05, 0.05, size=(3, 3))
    return _molecule(["O", "H", "H"], xyz, per, case["ng0"])


def _noisy_eris(n, seed):
    """ERIs of a positive metric with the spread eigenvalues of a real one, plus Monte Carlo noise
    that makes the small ones negative; in the order of build_mapping."""
    rng = np.random.default_rng(7919 * seed + 5)
    N = n * (n + 1) // 2
    Q, _ = np.linalg.qr(rng.standard_normal((N, N)))
    noise = rng.standard_normal((N, N)) * 1e-6
    M = (Q * 10.0 ** (1.0 - 7.0 * np.arange(N) / N)) @ Q.T + (noise + noise.T) / 2
    p, q = _pairs(n)
    return M[p, q]


def _pairs(n):
    i, j, k, l = [np.asarray(a, np.int64) - 1 for a in basis.build_mapping(n)]
    return i * (i + 1) // 2 + k, j * (j + 1) // 2 + l


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind, "seed": seed % (1 << 31)}
    if kind == "batch":
        rng = np.random.default_rng(1000003 * seed + 29)
        st["systems"] = [_mol(a, case["ng0"], rng)[1] for a in case["systems"].split("|")]
        st["seeds"] = [int(x) for x in rng.integers(1, 1 << 31, len(st["systems"]))]
        return st
    st["ctx"] = ctx = api.Context(0)
    if kind in ("svd", "project"):
        zetas = 0.8 + 0.05 * np.arange(case["n"])  # the basis only fixes n here
        _, b = _molecule(["H"], [[0.0, 0.0, 0.0]], {1: [("1S", float(z)) for z in zetas]}, 3)
        ctx.set_basis(b)
        ctx.set_quartets(*basis.build_mapping(b.n))
        st["moy"] = _noisy_eris(case["n"], seed)
        return st
    mol, b = _system(case, seed)
    st["basis"], st["quartets"] = b, basis.build_mapping(b.n)
    if kind == "one_e":
        st["xyz"], st["charge"] = mol.coords, mol.charges
    if kind == "mc":
        ctx.set_basis(b)
        ctx.set_quartets(*st["quartets"])
    return st


# ---- one pass --------------------------------------------------------------------------------
def run(st):
    case, kind = st["case"], st["kind"]
    if kind == "batch":
        res, _ = batch.batch_two_e(st["systems"], st["seeds"], sigma_target=0.0, npts=case["npts"],
                                   nblocks_max=case["nblocks"], a_zv=A_ZV)
        return res
    ctx = st["ctx"]
    if kind == "svd":
        moy, removed = ctx.psd_clean(st["moy"], layout=case["layout"], rank=case["rank"],
                                     oversample=case["oversample"], q=case["q"], seed=1)
        return {"eri": moy, "removed": removed}
    if kind == "project":
        moy, removed = ctx.psd_project(st["moy"], layout=case["layout"])
        return {"eri": moy, "removed": removed}
    if kind == "mc":
        mean, sigma = ctx.zvmc(A_ZV, st["seed"], case["npts"], case["nblocks"], case["estimator"], case["precision"])
        return {"mean": mean, "sigma": sigma}
    ctx.set_basis(st["basis"])
    if kind == "one_e":
        ctx.set_nuclei(st["xyz"], st["charge"])
        S, V, K = ctx.one_e()
        return {"S": S, "V": V, "K": K}
    ctx.set_quartets(*st["quartets"])
    if kind == "job":
        eri, sigma = ctx.two_e_job(A_ZV, st["seed"], case["npts"], case["nblocks"])
        return {"eri": eri, "sigma": sigma}
    eri, removed = ctx.gauss_eri()
    return {"eri": eri, "removed": removed}


# ---- the work of one pass --------------------------------------------------------------------
def _eri_work(b):
    """Analytic stage: a Boys evaluation and the Hermite integrals of every primitive quartet of
    every shell quartet (the components of a shell share them), and one multiply-add per unique
    integral and primitive quartet.  Half of the primitive quartets, about what screening keeps."""
    sh, first = np.unique(np.asarray(b.shell), return_index=True)
    deg = [2 if b.i_type[f] == 2 else int(b.npower[f].sum()) for f in first]
    ncomp = [int((np.asarray(b.shell) == s).sum()) for s in sh]
    ng = [int(b.n_gauss[f]) for f in first]
    pairs = []
    for x in range(len(sh)):
        for y in range(x + 1):
            same = x == y
            pairs.append((deg[x] + deg[y], ng[x] * (ng[x] + 1) // 2 if same else ng[x] * ng[y],
                          ncomp[x] * (ncomp[x] + 1) // 2 if same else ncomp[x] * ncomp[y]))
    d, p, c = (np.array(v, float) for v in zip(*pairs))
    L = d[:, None] + d[None, :]
    each = 30.0 + 2.0 * (L + 1) * (L + 2) * (L + 3) / 6.0 + 2.0 * c[:, None] * c[None, :]
    flops = 0.5 * (np.triu(p[:, None] * p[None, :] * each)).sum()
    n = b.n
    nq = (n * (n + 1) // 2) * (n * (n + 1) // 2 + 1) // 2
    return {"bytes": 8.0 * nq + 16.0 * nq + 16.0 * sum(ng), "flops": float(flops)}


def _mc_work(n, S, estimator):
    P = n * (n + 1) // 2
    nq = P * (P + 1) // 2
    if estimator == "shared":  # three bf16 products of the two-term densities per pair of pairs
        return {"bytes": 16.0 * nq, "flops": 3.0 * 2.0 * 2.0 * P * P * S}
    return {"bytes": 16.0 * nq, "flops": 12.0 * nq * S}  # distance, two products, two sums


def _add(*w):
    return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ws = []
        for a in case["systems"].split("|"):
            b = _mol(a, case["ng0"], np.random.default_rng(0))[1]
            ws += [_eri_work(b), _mc_work(b.n, case["npts"] * case["nblocks"], "shared")]
        return _add(*ws)
    if kind in ("svd", "project"):
        N = case["n"] * (case["n"] + 1) // 2
        if kind == "project":  # tridiagonal reduction, eigenvectors, rank update
            return {"bytes": 16.0 * N * N, "flops": (4.0 / 3.0 + 4.0 + 2.0) * N ** 3}
        r = min(N, case["rank"] + case["oversample"])
        return {"bytes": 16.0 * N * N, "flops": 2.0 * N * N * r * (2 * case["q"] + 3) + 8.0 * N * r * r}
    b = _system(case, 0)[1]
    if kind == "eri":
        return _eri_work(b)
    if kind == "mc":
        return _mc_work(b.n, case["npts"] * case["nblocks"], case["estimator"])
    if kind == "job":
        return _add(_eri_work(b), _mc_work(b.n, case["npts"] * case["nblocks"], "shared"))
    prim = float(np.sum(b.n_gauss)) ** 2  # overlap, kinetic and one Boys evaluation per nucleus
    nat = len(set(np.asarray(b.nucleus).tolist()))
    return {"bytes": 8.0 * 3 * b.n ** 2 + 8.0 * b.n * (5 + 3 * b.ld), "flops": prim * (60.0 + 60.0 * nat)}


# ---- the same in plain 64-bit torch ----------------------------------------------------------
def _boys(m, T):
    """F_0..F_m(T): the ascending series and downward recursion for T < 40, erf and upward
    recursion above (stable there)."""
    small = T < 40.0
    Ts = torch.where(small, T, torch.zeros_like(T))
    e = torch.exp(-Ts)
    term = torch.full_like(Ts, 1.0 / (2 * m + 1))
    s = term.clone()
    for i in range(1, 180):
        term = term * (2.0 * Ts) / (2 * m + 2 * i + 1)
        s = s + term
    lo = [None] * (m + 1)
    lo[m] = s * e
    for n in range(m - 1, -1, -1):
        lo[n] = (2.0 * Ts * lo[n + 1] + e) / (2 * n + 1)
    Tb = torch.where(small, torch.full_like(T, 40.0), T)
    eb = torch.exp(-Tb)
    hi = [0.5 * torch.sqrt(math.pi / Tb) * torch.erf(torch.sqrt(Tb))]
    for n in range(m):
        hi.append(((2 * n + 1) * hi[n] - eb) / (2.0 * Tb))
    return [torch.where(small, a, b) for a, b in zip(lo, hi)]


def _hermite(L, alpha, R):
    """R_tuv (t + u + v <= L) of McMurchie and Davidson at exponent alpha and distance R."""
    F = _boys(L, alpha * (R[0] ** 2 + R[1] ** 2 + R[2] ** 2))
    cur = {(0, 0, 0): (-2.0 * alpha) ** L * F[L]}
    for m in range(L - 1, -1, -1):
        nxt = {(0, 0, 0): (-2.0 * alpha) ** m * F[m]}
        for tot in range(1, L - m + 1):
            for t in range(tot + 1):
                for u in range(tot - t + 1):
                    v = tot - t - u
                    ix = [t, u, v]
                    ax = next(a for a in range(3) if ix[a] > 0)
                    lo = list(ix)
                    lo[ax] -= 1
                    val = R[ax] * cur[tuple(lo)]
                    if lo[ax] > 0:
                        lo2 = list(lo)
                        lo2[ax] -= 1
                        val = val + lo[ax] * cur[tuple(lo2)]
                    nxt[(t, u, v)] = val
        cur = nxt
    return cur


def _E(i, j, PA, PB, p):
    """Hermite expansion coefficients E_t^{ij} along one axis (without the exponential)."""
    one = torch.ones_like(p)
    E = {(0, 0): [one]}

    def get(v, t):
        return v[t] if 0 <= t < len(v) else torch.zeros_like(p)

    def raise_(v, x):
        n = len(v)
        return [get(v, t - 1) / (2.0 * p) + x * get(v, t) + (t + 1) * get(v, t + 1) for t in range(n + 1)]

    for a in range(i):
        E[(a + 1, 0)] = raise_(E[(a, 0)], PA)
    for c in range(j):
        E[(i, c + 1)] = raise_(E[(i, c)], PB)
    return E[(i, j)]


class _Pair:
    """Primitive products of two functions, over all pairs of their exponents."""

    def __init__(self, b, i, k, dev):
        t = lambda x: torch.tensor(np.asarray(x, np.float64), device=dev)  # noqa: E731
        A, B = b.center[i], b.center[k]
        a = t(b.g_gauss[i, :b.n_gauss[i]])[:, None]
        c = t(b.g_gauss[k, :b.n_gauss[k]])[None, :]
        self.a, self.c = (x.reshape(-1) for x in torch.broadcast_tensors(a, c))
        self.p = self.a + self.c
        R2 = float(((A - B) ** 2).sum())
        self.P = [(self.a * float(A[x]) + self.c * float(B[x])) / self.p for x in range(3)]
        self.PA = [self.P[x] - float(A[x]) for x in range(3)]
        self.PB = [self.P[x] - float(B[x]) for x in range(3)]
        ci = t(b.c_gauss[b.i_type[i] - 1, i, :b.n_gauss[i]])[:, None]
        ck = t(b.c_gauss[b.i_type[k] - 1, k, :b.n_gauss[k]])[None, :]
        self.w = (ci * ck).reshape(-1) * torch.exp(-self.a * self.c / self.p * R2)


def _comps(b, f):
    """Cartesian powers whose sum is the function (the r^2-type fits are x^2 + y^2 + z^2)."""
    if b.i_type[f] == 2:
        return [tuple(int(v) + (2 if a == x else 0) for a, v in enumerate(b.npower[f])) for x in range(3)]
    return [tuple(int(v) for v in b.npower[f])]


def _density(b, i, k, P):
    """{(t, u, v): coefficient} of the charge distribution of functions i and k."""
    out = {}
    for ci in _comps(b, i):
        for ck in _comps(b, k):
            ex = [_E(ci[x], ck[x], P.PA[x], P.PB[x], P.p) for x in range(3)]
            for t, et in enumerate(ex[0]):
                for u, eu in enumerate(ex[1]):
                    for v, ev in enumerate(ex[2]):
                        val = P.w * et * eu * ev
                        out[(t, u, v)] = out[(t, u, v)] + val if (t, u, v) in out else val
    return out


def _exact_eri(b):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = b.n
    first = {int(s): int(np.nonzero(np.asarray(b.shell) == s)[0][0]) for s in np.unique(b.shell)}
    pp, dens, deg = {}, {}, {}
    for i in range(n):
        for k in range(i + 1):
            key = (int(b.shell[i]), int(b.shell[k]))
            if key not in pp:
                pp[key] = _Pair(b, first[key[0]], first[key[1]], dev)
            d = _density(b, i, k, pp[key])
            # Hermite terms along the ket carry the sign (-1)^(t+u+v)
            dens[(i, k)] = {h: v for h, v in d.items() if bool((v != 0).any())}
            deg[key] = max(deg.get(key, 0), max((sum(h) for h in dens[(i, k)]), default=0))
    i_, j_, k_, l_ = [np.asarray(a) - 1 for a in basis.build_mapping(n)]
    groups = {}
    for q in range(len(i_)):
        a, c = (int(i_[q]), int(k_[q])), (int(j_[q]), int(l_[q]))
        if a[0] < c[0] or (a[0] == c[0] and a[1] < c[1]):
            a, c = c, a
        key = tuple((int(b.shell[x]), int(b.shell[y])) for x, y in (a, c))
        groups.setdefault(key, {}).setdefault(c, {}).setdefault(a, []).append(q)
    out = torch.zeros(len(i_), dtype=torch.float64, device=dev)
    for (kb, kk), kets in groups.items():
        P, Q = pp[kb], pp[kk]
        p, s = P.p[:, None], Q.p[None, :]
        alpha = p * s / (p + s)
        R = _hermite(deg[kb] + deg[kk], alpha, [P.P[x][:, None] - Q.P[x][None, :] for x in range(3)])
        pre = 2.0 * math.pi ** 2.5 / (p * s * torch.sqrt(p + s))
        R = {h: v * pre for h, v in R.items()}
        for c, bras in kets.items():
            need = sorted({h for a in bras for h in dens[a]})
            col = {}
            for h in need:
                g = torch.zeros_like(P.p)
                for h2, e in dens[c].items():
                    g = g + (-1.0) ** sum(h2) * (R[tuple(x + y for x, y in zip(h, h2))] @ e)
                col[h] = g
            for a, qs in bras.items():
                v = sum((dens[a][h] * col[h]).sum() for h in dens[a])
                for q in qs:
                    out[q] = v
    return out.cpu().numpy()


def _exact_one_e(b, xyz, charge):
    n = b.n
    S, V, K = (np.zeros((n, n)) for _ in range(3))
    for i in range(n):
        for k in range(n):
            P = _Pair(b, i, k, "cpu")
            d = _density(b, i, k, P)
            S[i, k] = float((d[(0, 0, 0)] * (math.pi / P.p) ** 1.5).sum())
            L = max(sum(h) for h in d)
            for at in range(len(charge)):
                R = _hermite(L, P.p, [P.P[x] - float(xyz[at][x]) for x in range(3)])
                V[i, k] -= charge[at] * float(sum((2.0 * math.pi / P.p * d[h] * R[h]).sum() for h in d))
            kin = torch.zeros_like(P.p)
            ov = (math.pi / P.p) ** 1.5 * P.w
            for ci in _comps(b, i):
                for ck in _comps(b, k):
                    s = lambda x, j: _E(ci[x], j, P.PA[x], P.PB[x], P.p)[0] if j >= 0 else 0.0  # noqa: E731
                    for x in range(3):
                        j = ck[x]
                        t = -2.0 * P.c ** 2 * s(x, j + 2) + P.c * (2 * j + 1) * s(x, j) - 0.5 * j * (j - 1) * s(x, j - 2)
                        y, z = (x + 1) % 3, (x + 2) % 3
                        kin = kin + t * s(y, ck[y]) * s(z, ck[z])
            K[i, k] = float((kin * ov).sum())
    return {"S": S, "V": V, "K": K}


def exact(case, seed):
    kind = case["kind"]
    if kind == "eri":
        b = _system(case, seed)[1]
        if b.n > 11:
            return None
        return {"eri": _exact_eri(b), "removed": None}
    if kind == "one_e":
        mol, b = _system(case, seed)
        return _exact_one_e(b, mol.coords, mol.charges)
    if kind == "project":
        n = case["n"]
        p, q = _pairs(n)
        N = n * (n + 1) // 2
        M = np.zeros((N, N))
        M[p, q] = M[q, p] = _noisy_eris(n, seed)
        lam, U = np.linalg.eigh(M)
        return {"eri": ((U * np.maximum(lam, 0.0)) @ U.T)[p, q], "removed": None}
    return None
