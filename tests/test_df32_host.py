"""Two-float arithmetic (csrc/df32.cuh) and the Boys functions of the shell-quartet kernels
(csrc/shell_eri.cuh) on the host, against exact rationals and 40-digit mpmath values.

Tolerances.  Two floats with |l| <= 2^-24 |h|: a product drops l l' (2^-48) and rounds its low part
twice at 2^-24 of at most 3 x 2^-24, together below 2^-45; a sum rounds its low part twice, below
2^-46 of |a| + |b|; the root's residual is a few roundings of 2^-24 at 2^-24, below 2^-45; the
three-part difference rounds its low parts three times, below 2^-46 of itself plus 2^-70 of the
coordinates.  F_m: the Taylor series and at most 8 recursion steps of three operations each, and in two
floats the tail of the series in FP32 (1e-8 x 2^-24): 30 x 2^-45 = 1e-12 / 1.2; in FP64 30 x 2^-53 with
the 2-ulp exponential, 5e-15; in FP32 30 x 2^-24 with T itself rounded, 4e-6."""
import ctypes as C
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

import eri_host

mp = pytest.importorskip("mpmath")
pytestmark = pytest.mark.skipif(not eri_host.available(), reason="needs g++ and the CUDA headers")

f32p = np.ctypeslib.ndpointer(np.float32, flags="C")
f64p = np.ctypeslib.ndpointer(np.float64, flags="C")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = Path(shutil.which("nvcc")).resolve().parent.parent / "include"
    out = tmp_path_factory.mktemp("df32") / "libdf32.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC", f"-I{inc}",
                    str(eri_host.HERE / "df32_host_shim.cpp"), "-o", str(out)], check=True)
    L = C.CDLL(str(out))
    L.ss_host_df.argtypes = [C.c_int, C.c_int, f32p, f32p, f32p, f32p]
    L.ss_host_shell_boys.argtypes = [C.c_int, C.c_int, f64p, f64p, f64p, f64p]
    return L


def _two(x):
    h = x.astype(np.float32)
    return np.stack([h, (x - h.astype(np.float64)).astype(np.float32)], axis=-1)


def _exact(a):
    return [sum(Fraction(float(v)) for v in row) for row in a]


def _call(L, op, a, b=None, c=None):
    out = np.zeros((len(a), 2), np.float32)
    z = np.zeros((1, 3), np.float32)
    L.ss_host_df(op, len(a), *[np.ascontiguousarray(z if x is None else x) for x in (a, b, c)], out)
    return _exact(out)


@pytest.fixture(scope="module")
def values():
    rng = np.random.default_rng(4)
    draw = lambda: rng.standard_normal(4000) * 10.0 ** rng.uniform(-6, 6, 4000)  # noqa: E731
    return _two(draw()), _two(draw()), _two(draw())


def test_sum_product_fma(lib, values):
    a, b, c = values
    ea, eb, ec = (_exact(v) for v in values)
    for x, y, r in zip(ea, eb, _call(lib, 0, a, b)):
        assert abs(r - (x + y)) <= Fraction(1, 2 ** 46) * (abs(x) + abs(y))
    for x, y, r in zip(ea, eb, _call(lib, 1, a, b)):
        assert abs(r - x * y) <= Fraction(1, 2 ** 45) * abs(x * y)
    for x, y, z, r in zip(ea, eb, ec, _call(lib, 2, a, b, c)):
        assert abs(r - (x * y + z)) <= Fraction(1, 2 ** 45) * abs(x * y) + Fraction(1, 2 ** 46) * (abs(x * y) + abs(z))


def test_reciprocal_root(lib, values):
    a = np.where(values[0][:, :1] < 0, -values[0], values[0])
    mp.mp.dps = 40
    for x, r in zip(_exact(a), _call(lib, 3, a)):
        want = 1 / mp.sqrt(mp.mpf(x.numerator) / x.denominator)
        assert abs((mp.mpf(r.numerator) / r.denominator) / want - 1) <= mp.mpf(2) ** -45


@pytest.mark.parametrize("apart", [1.0, 1e-3, 1e-7, 1e-12])
def test_difference_of_three_parts(lib, apart):
    rng = np.random.default_rng(7)
    x = rng.uniform(-200.0, 200.0, 3000)
    y = x + apart * rng.standard_normal(3000)

    def three(v):
        h = v.astype(np.float32)
        m = (v - h).astype(np.float32)
        return np.stack([h, m, (v - h - m).astype(np.float32)], axis=-1)

    a, b = three(x), three(y)
    for u, v, r in zip(_exact(a), _exact(b), _call(lib, 4, a, b)):
        assert abs(r - (u - v)) <= Fraction(1, 2 ** 46) * abs(u - v) + Fraction(200, 2 ** 70)


@pytest.mark.parametrize("L", [0, 1, 4, 8])
def test_boys_functions(lib, L):
    rng = np.random.default_rng(L)
    edges = [x + d for x in (0.0625, 1.0, 29.9375, 30.0, 36.0, 80.0) for d in (-1e-7, -1e-12, 0.0, 1e-12, 1e-7)]
    T = np.array([0.0, 1e-300, 1e-12] + edges + list(rng.uniform(0, 40, 150)) + list(10.0 ** rng.uniform(-6, 4, 80)))
    out = [np.zeros((len(T), 9)) for _ in range(3)]
    assert lib.ss_host_shell_boys(L, len(T), T, *out) == 0
    mp.mp.dps = 40
    for i, t in enumerate(T):
        for m in range(L + 1):
            x = mp.mpf(float(t))
            want = (mp.mpf(1) / (2 * m + 1) if t < 1e-30
                    else mp.gammainc(m + mp.mpf(1) / 2, 0, x) / (2 * x ** (m + mp.mpf(1) / 2)))
            tiny = want < 1e-36  # below FP32's normal range: the FP32 results may underflow
            for got, tol in zip(out, (5e-15, 1e-12 / 1.2, 4e-6)):
                if tol > 1e-14 and tiny:
                    continue
                assert abs(mp.mpf(float(got[i, m])) / want - 1) <= tol, (t, m, tol)
