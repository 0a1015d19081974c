"""Sizes of the shell-pair tables (csrc/shell_basis.h, host build): pairs of one system only, and room
for the primitives that survive the K_AB screen, not for all products."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import eri_host
from slater_stoch_gb300 import basis, batch, configs

pytestmark = pytest.mark.skipif(not eri_host.available(), reason="needs g++ and the CUDA headers")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = Path(shutil.which("nvcc")).resolve().parent.parent / "include"
    out = tmp_path_factory.mktemp("shells") / "libshells.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{inc}",
                    str(eri_host.HERE / "shell_host_shim.cpp"), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def _tables(L, b, first=None):
    center, npower, _, i_type, n_gauss, c_gauss, g_gauss, _ = eri_host.basis_arrays(b)
    sys = None
    if first is not None:
        sys = np.repeat(np.arange(len(first) - 1, dtype=np.int32), np.diff(first))
    cap, fa, fb = (np.zeros(1 << 16, np.int32) for _ in range(3))
    out, fn = np.zeros(4, np.int64), np.zeros((b.n, b.n), np.int32)
    p = lambda a: None if a is None else a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rc = L.ss_host_shells(int(b.n), int(b.ld), p(center), p(npower), p(i_type), p(n_gauss), p(c_gauss), p(g_gauss), p(sys),
                          p(out), len(cap), p(cap), p(fa), p(fb), p(fn))
    assert rc == 0
    n = int(out[1])
    return {"shells": int(out[0]), "pairs": n, "prims": int(out[2]), "coefs": int(out[3]), "cap": cap[:n], "fa": fa[:n],
            "fb": fb[:n], "fn": fn}


def _atoms(count, seed=3):
    rng = np.random.default_rng(seed)
    return [configs.random_molecule(int(rng.integers(1, 2 ** 31 - 1)), natoms=1, box=4.0, ng0=6) for _ in range(count)]


def test_a_batch_holds_the_tables_of_its_systems(lib):
    systems = _atoms(40)
    comb, first = batch.concat_systems(systems)
    t = _tables(lib, comb, first)
    alone = [_tables(lib, b) for b in systems]
    for key in ("shells", "pairs", "prims", "coefs"):
        assert t[key] == sum(a[key] for a in alone)
    sys = np.repeat(np.arange(len(systems)), np.diff(first))
    i, k = np.tril_indices(comb.n)
    assert np.array_equal(t["fn"][i, k] >= 0, sys[i] == sys[k])


@pytest.mark.parametrize("dist", [0.7, 3.0, 12.0, 60.0])
def test_room_follows_the_screen(lib, dist):
    """Never fewer places than primitives that the device keeps, and no more than 2 % above them."""
    mol = basis.molecule_bohr(["O", "C"], [[0.1, -0.2, 0.3], [0.1 + dist, 0.1, 0.2]])
    orbs = [("1S", 7.7), ("2S", 2.2), ("2P", 2.1), ("3D", 1.3)]
    b = basis.build_basis(mol, {8: orbs, 6: orbs}, basis.FitParams(ng0=20))
    t = _tables(lib, b)
    for cap, f, g in zip(t["cap"], t["fa"], t["fb"]):
        a, c = b.g_gauss[f, :b.n_gauss[f], None], b.g_gauss[g, None, :b.n_gauss[g]]
        r2 = float(((b.center[f] - b.center[g]) ** 2).sum())
        kk = a * c / (a + c) * r2
        keep = (kk <= 40.0) & (np.exp(-kk) >= 1e-15)
        n = int(keep.sum())
        if r2 == 0.0:
            assert cap == (b.n_gauss[f] * (b.n_gauss[f] + 1) // 2 if f == g else n)
        else:
            assert n <= cap <= n + max(1, n // 50)
