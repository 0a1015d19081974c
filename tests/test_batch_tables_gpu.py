"""Batches of many systems under a device-memory budget: the analytic tables are those of the systems,
not of every two of them, and each system's values equal, bit for bit, the system alone."""
import numpy as np
import pytest

from slater_stoch_gb300 import api, basis, batch, configs
from slater_stoch_gb300._lib import check

pytestmark = pytest.mark.gpu


def _atom(symbol, rng):
    z = basis.element_number(symbol)
    orbs = ("1S", "2P") if z == 1 else ("1S", "2S", "2P", "3D")
    mol = basis.molecule_bohr([symbol], rng.uniform(-2.0, 2.0, (1, 3)))
    return basis.build_basis(mol, {z: [(o, configs.SLATER[z][o] * rng.uniform(0.8, 1.2)) for o in orbs]},
                             basis.FitParams(ng0=20))


@pytest.mark.parametrize("symbols,count,budget", [("HCNO", 64, 1 << 30), ("H", 512, 1 << 30)])
def test_many_systems_fit_a_budget(symbols, count, budget):
    rng = np.random.default_rng(count)
    systems = [_atom(symbols[s % len(symbols)], rng) for s in range(count)]
    comb, first = batch.concat_systems(systems)
    lists = [[np.asarray(a, np.int32) for a in basis.build_mapping(b.n)] for b in systems]
    cat = [np.ascontiguousarray(np.concatenate([q[c] + (int(f) - 1) for q, f in zip(lists, first)])) for c in range(4)]
    with api.Context(0, budget) as ctx:
        ctx.set_basis(comb)
        check(ctx._L.ss_basis_systems(ctx._h, count, first))
        ctx.set_quartets(*cat)
        together, _ = ctx.gauss_eri()
        pre = ctx.precond()
    sys = np.repeat(np.arange(count), np.diff(first))
    assert np.all(pre[sys[:, None] != sys[None, :]] == 0.0)
    offs = np.cumsum([0] + [len(q[0]) for q in lists])
    for s in range(0, count, max(1, count // 12)):
        with api.Context(0) as ctx:
            ctx.set_basis(systems[s])
            ctx.set_quartets(*lists[s])
            np.testing.assert_array_equal(together[offs[s]:offs[s + 1]], ctx.gauss_eri()[0])
