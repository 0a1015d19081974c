"""Faithful ZV-MC estimator at the edges of its pair groups and quartet tiles: functions of several
shells in mixed order with components missing, bra pairs with 1 to many quartets, walker counts
that are no multiple of a warp.  The oracle evaluates the same walkers.

The shared estimator's operand kernel at several pairs per CTA (2 and 8, the last CTA with a
remainder) and sample counts that are no multiple of its vectors.

Gate (faithful): |dmean| <= 1e-10 |ERI| + 1e-13 sqrt((ik|ik)(jl|jl)), 1e-9 for ref32.  A sum of up to 280
weighted terms rounds at about 300 2^-53 = 3e-14 of their mean magnitude, a few Schwarz bounds.
"""
import dataclasses

import numpy as np
import pytest

from slater_stoch_gb300 import api, basis

pytestmark = pytest.mark.gpu


def _mixed_basis():
    mol = basis.molecule_bohr(["O", "C"], [[0.1, -0.2, 0.3], [1.3, 0.9, -1.1]])
    per = {z: [(o, 1.1 + 0.7 * t) for t, o in enumerate(["1S", "2S", "2P", "3D"])] for z in (8, 6)}
    b = basis.build_basis(mol, per, basis.FitParams(ng0=4))
    order = np.random.default_rng(5).permutation(b.n)[: b.n - 5]
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


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-10), ("ref32", 1e-9)])
@pytest.mark.parametrize("npts,count", [(80, 40), (40, 1500), (280, 1500), (40, 11000)])
def test_pair_groups_and_tiles(npts, count, precision, rtol):
    from oracle import binding as O
    b = _mixed_basis()
    full = basis.build_mapping(b.n)
    pick = np.sort(np.random.default_rng(count).choice(len(full[0]), count, replace=False))
    q = tuple(np.asarray(a)[pick] for a in full)
    nblocks = 3
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        r1, r2 = ctx.draw_walkers(seed=5, first=0, S=nblocks * npts)
        mean, _ = ctx.zvmc_walkers(1.8, r1, r2, npts, nblocks, precision)
    O.set_sum_mode("extended")
    ob = O.OracleBasis(b)
    ref, _ = O.zvmc_faithful(ob, q, 1.8, r1, r2, nblocks, npts, precision)
    flat = O.precond(ob)
    gauss = O.gauss_eri(ob, q, flat)[0]
    pre = flat.reshape(b.n, b.n, order="F")
    i, j, k, l = [np.asarray(a) - 1 for a in q]
    bound = rtol * np.abs(gauss + ref) + 1e-13 * np.sqrt(np.abs(pre[i, k] * pre[j, l]))
    d = np.abs(mean - ref)
    assert np.all(d <= bound), float(np.max(d / bound))


@pytest.mark.parametrize("npts", [70001, 250001])
def test_shared_pairs_per_cta(npts):
    """Gate: 1e-5 sqrt((ik|ik)(jl|jl)).  The split-BF16 products drop 2^-16 of their terms, and the
    terms of the correction are about 1e-2 of the Schwarz bound with 4-Gaussian fits; a wrong pair or
    sample shows at that 1e-2."""
    from oracle import binding as O
    b = _mixed_basis()
    full = basis.build_mapping(b.n)
    pick = np.sort(np.random.default_rng(9).choice(len(full[0]), 1500, replace=False))
    q = tuple(np.asarray(a)[pick] for a in full)
    nblocks = 2
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        mean, _ = ctx.zvmc(a_zv=1.8, seed=13, npts=npts, nblocks=nblocks, estimator="shared", precision="split_bf16")
        u1, u2, w = ctx.shared_samples(1.8, seed=13, first=0, S=nblocks * npts)
    O.set_sum_mode("extended")
    ob = O.OracleBasis(b)
    ref, _ = O.zvmc_shared(ob, q, u1, u2, w, nblocks, npts, symmetrize=True)
    pre = O.precond(ob).reshape(b.n, b.n, order="F")
    i, j, k, l = [np.asarray(a) - 1 for a in q]
    bound = 1e-5 * np.sqrt(np.abs(pre[i, k] * pre[j, l]))
    d = np.abs(mean - ref)
    assert np.all(d <= bound), float(np.max(d / bound))
