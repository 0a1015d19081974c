"""The shell-quartet ERI kernel (csrc/shell_eri.cuh) at the edges of its dispatch: every pair type
on one and two centres, fits of 1 to 30 Gaussians (one primitive, partly filled and many bra
slices), shells that lack components, functions of several shells in mixed order, functions in no
shell beside functions in shells, and lists that ask for a few members of a shell quartet.

Gate per quartet, as for the other analytic ERIs: 1e-12 |ERI| + 1e-12 sqrt((ik|ik)(jl|jl)).
"""
import dataclasses

import numpy as np
import pytest

from slater_stoch_gb300 import api, basis, configs

pytestmark = pytest.mark.gpu

XYZ = [[0.1, -0.2, 0.3], [1.3, 0.9, -1.1]]


def _basis(orbs, ng0, atoms=2):
    mol = basis.molecule_bohr(["O", "C"][:atoms], XYZ[:atoms])
    per = {8: [(o, 1.1 + 0.7 * t) for t, o in enumerate(orbs)], 6: [(o, 0.8 + 0.6 * t) for t, o in enumerate(orbs)]}
    return basis.build_basis(mol, per, basis.FitParams(ng0=ng0))


def _take(b, order):
    f = {}
    for fld in dataclasses.fields(b):
        v = getattr(b, fld.name)
        if fld.name == "c_gauss":
            f[fld.name] = np.ascontiguousarray(v[:, order])
        elif fld.name == "names":
            f[fld.name] = [v[i] for i in order]
        else:
            f[fld.name] = np.ascontiguousarray(v[order])
    return basis.Basis(**f)


def _compare(b, q):
    from oracle import binding as O
    O.set_sum_mode("extended")
    ob = O.OracleBasis(b)
    pre = O.precond(ob)
    ref, nz_ref = O.gauss_eri(ob, q, pre)
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        gp = ctx.precond()
        g, nz = ctx.gauss_eri()
    np.testing.assert_allclose(gp.reshape(-1, order="F"), pre, rtol=1e-12, atol=0)
    assert nz == nz_ref
    P = pre.reshape(b.n, b.n, order="F")
    i, j, k, l = [np.asarray(a) - 1 for a in q]
    bound = 1e-12 * np.abs(ref) + 1e-12 * np.sqrt(np.abs(P[i, k] * P[j, l]))
    assert np.all(np.abs(g - ref) <= bound), float(np.max(np.abs(g - ref) / np.maximum(bound, 1e-300)))
    return g


def _sample(n, count, seed=1):
    q = [np.asarray(a) for a in basis.build_mapping(n)]
    if len(q[0]) <= count:
        return q
    sel = np.sort(np.random.default_rng(seed).choice(len(q[0]), count, replace=False))
    return [np.ascontiguousarray(a[sel]) for a in q]


@pytest.mark.parametrize("atoms", [1, 2])
@pytest.mark.parametrize("ng0", [1, 2, 3])
def test_all_pair_types(atoms, ng0):
    b = _basis(["1S", "2S", "2P", "3D"], ng0, atoms)
    _compare(b, _sample(b.n, 6000))


@pytest.mark.parametrize("orbs,ng0,count", [(["1S"], 30, 10), (["1S", "2S"], 9, 25), (["2P"], 30, 40), (["3D"], 6, 500)])
def test_fit_lengths(orbs, ng0, count):
    b = _basis(orbs, ng0)
    _compare(b, _sample(b.n, count))


def test_partial_shells_in_mixed_order():
    b = _basis(["1S", "2S", "2P", "3D"], 2)
    order = np.random.default_rng(3).permutation(b.n)[: b.n - 7]
    _compare(_take(b, order), _sample(b.n - 7, 6000))


def test_function_in_no_shell():
    """x y z times a Gaussian fit (degree 3) takes the per-function kernels, its neighbours too where
    they meet it in a quartet."""
    b = _basis(["1S", "2S", "2P"], 2)
    b.npower[2] = [1, 1, 1]
    b.npower[7] = [1, 1, 1]
    _compare(b, _sample(b.n, 3000))


def test_a_value_does_not_depend_on_the_list():
    b = _basis(["1S", "2S", "2P", "3D"], 4)
    q = [np.asarray(a) for a in basis.build_mapping(b.n)]
    sel = np.random.default_rng(5).choice(len(q[0]), 300, replace=False)
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        full, _ = ctx.gauss_eri()
        ctx.set_quartets(*[np.ascontiguousarray(a[sel]) for a in q])
        some, _ = ctx.gauss_eri()
        np.testing.assert_array_equal(some, full[sel])
        ctx.set_quartets(*[np.ascontiguousarray(a[sel[:1]]) for a in q])
        one, _ = ctx.gauss_eri()
        np.testing.assert_array_equal(one, full[sel[:1]])


def test_all_fp64_tier():
    """fp32_eps <= screen_eps evaluates every kept primitive quartet in FP64, screen_eps = 0 keeps all."""
    b = configs.h2o_minimal(ng0=6)
    q = basis.build_mapping(b.n)
    from oracle import binding as O
    O.set_sum_mode("extended")
    ob = O.OracleBasis(b)
    pre = O.precond(ob)
    ref, _ = O.gauss_eri(ob, q, pre)
    P = pre.reshape(b.n, b.n, order="F")
    i, j, k, l = [np.asarray(a) - 1 for a in q]
    bound = 1e-12 * np.abs(ref) + 1e-12 * np.sqrt(np.abs(P[i, k] * P[j, l]))
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        for screen, fp32 in ((1e-18, 0.0), (0.0, 0.0), (0.0, 1e-11)):
            ctx.set_eri_tiers(screen, fp32)
            g, _ = ctx.gauss_eri()
            assert np.all(np.abs(g - ref) <= bound)
