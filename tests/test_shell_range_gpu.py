"""The two-float and FP32 tiers of the shell-quartet ERIs where FP32's range or digits could be left:
fits of 30 Gaussians (exponents over 8 decades and more), exponents that differ between the shells,
one and two centres, a molecule far from the origin.  Every value against the same kernels with the tiers off (all FP64), and a sample
against the oracle.

Gate per quartet, as for the other analytic ERIs: 1e-12 |ERI| + 1e-12 sqrt((ik|ik)(jl|jl)).
"""
import numpy as np
import pytest

from slater_stoch_gb300 import api, basis

pytestmark = pytest.mark.gpu

ONE = [[0.1, -0.2, 0.3]]
TWO = ONE + [[1.3, 0.9, -1.1]]
ORBS = {"d": [("3D", 3.0)], "tight_d": [("3D", 1.0), ("3D", 10.0)], "tight_s": [("2S", 0.5), ("2S", 20.0), ("2P", 10.0)],
        "mixed": [("1S", 50.0), ("2P", 20.0), ("2P", 0.5), ("3D", 1.0)]}


def _basis(orbs, ng0, xyz):
    mol = basis.molecule_bohr(["O", "C"][:len(xyz)], xyz)
    return basis.build_basis(mol, {8: orbs, 6: orbs}, basis.FitParams(ng0=ng0))


def _gate(value, ref, pre, q):
    i, j, k, l = [np.asarray(a) - 1 for a in q]
    bound = 1e-12 * np.abs(ref) + 1e-12 * np.sqrt(np.abs(pre[i, k] * pre[j, l]))
    d = np.abs(value - ref)
    assert np.all(d <= bound), float(np.max(d / np.maximum(bound, 1e-300)))


def _default_and_fp64(b, q):
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        pre = ctx.precond()
        g, _ = ctx.gauss_eri()
        ctx.set_eri_tiers(1e-18, 0.0)
        f, _ = ctx.gauss_eri()
    return g, f, pre


@pytest.mark.parametrize("ng0", [20, 30])
@pytest.mark.parametrize("xyz", [ONE, TWO], ids=["one_centre", "two_centres"])
@pytest.mark.parametrize("orbs", list(ORBS))
def test_tiers_against_fp64(orbs, xyz, ng0):
    b = _basis(ORBS[orbs], ng0, xyz)
    q = basis.build_mapping(b.n)
    g, f, pre = _default_and_fp64(b, q)
    _gate(g, f, pre, q)


@pytest.mark.parametrize("orbs", ["d", "tight_s"])
def test_long_fits_against_the_oracle(orbs):
    from oracle import binding as O
    O.set_sum_mode("extended")
    b = _basis(ORBS[orbs], 30, TWO)
    full = [np.asarray(a) for a in basis.build_mapping(b.n)]
    pick = np.sort(np.random.default_rng(2).choice(len(full[0]), 30, replace=False))
    q = [np.ascontiguousarray(a[pick]) for a in full]
    ob = O.OracleBasis(b)
    ref, _ = O.gauss_eri(ob, q, O.precond(ob))
    g, _, pre = _default_and_fp64(b, q)
    _gate(g, ref, pre, q)


@pytest.mark.parametrize("orbs", list(ORBS))
def test_far_from_the_origin(orbs):
    b = _basis(ORBS[orbs], 20, [[100.1, -60.2, 33.3], [101.3, -59.1, 32.2]])
    q = basis.build_mapping(b.n)
    g, f, pre = _default_and_fp64(b, q)
    _gate(g, f, pre, q)


def test_tiers_without_a_screen():
    """screen_eps = 0 skips nothing and leaves the other thresholds as they are: the same values as with a
    screen below every primitive quartet's bound, and not those of the all-FP64 evaluation."""
    b = _basis(ORBS["mixed"], 12, TWO)
    q = basis.build_mapping(b.n)
    out = {}
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        pre = ctx.precond()
        for screen, fp32 in ((0.0, 1e-11), (1e-300, 1e-11), (0.0, 0.0)):
            ctx.set_eri_tiers(screen, fp32)
            out[screen, fp32], _ = ctx.gauss_eri()
    np.testing.assert_array_equal(out[0.0, 1e-11], out[1e-300, 1e-11])
    assert not np.array_equal(out[0.0, 1e-11], out[0.0, 0.0])
    _gate(out[0.0, 1e-11], out[0.0, 0.0], pre, q)
