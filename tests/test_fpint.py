"""The integer-pipe FP64 operations of the device (csrc/fpint.h), built for the host:
division, square root, rounding and comparison against NumPy's FP64 arithmetic, and
detmath.h's functions on top of them against the oracle's plain build, all bit for
bit, at the edges of each operation's range and with the approximate reciprocals moved
by their error bound."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import _oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "etraj.jl_gb300", "csrc")
N = 200000


@pytest.fixture(scope="module")
def fp(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fpint") / "libfpint.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math",
                    "-I" + CSRC, os.path.join(HERE, "fpint_probe.cpp"), "-o", out], check=True)
    lib = C.CDLL(out)
    DP = C.POINTER(C.c_double)
    lib.fp_op.argtypes = [C.c_int, C.c_long, DP, DP, DP]
    lib.fp_set_ulp.argtypes = [C.c_double]

    def call(op, x, y=None):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.ascontiguousarray(x if y is None else y, dtype=np.float64)
        r = np.zeros_like(x)
        lib.fp_op(op, x.size, x.ctypes.data_as(DP), y.ctypes.data_as(DP), r.ctypes.data_as(DP))
        return r

    call.set_ulp = lib.fp_set_ulp
    yield call
    lib.fp_set_ulp(0.0)


SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, 2.0, 4.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                    1.7976931348623157e308, np.nextafter(1.0, 0), np.nextafter(1.0, 2), np.nextafter(2.0, 0),
                    np.nextafter(4.0, 0), 1e-300, 1e300, 3.0, 0.5, 60.0, 22.0, 38.0, -38.0, 708.0, -708.0, 709.9, -745.2,
                    1e-9, 1.4142135623730951, 262144.0, -262144.0, 1e10])


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64)) or \
        bool(np.all((a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))))


def mantissas(rng, n):
    """Mantissas with long runs of ones and zeros among random ones, exponents over the range."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = np.arange(n) % 5
    m[k == 1] |= np.uint64(0xFFFFFFFFFF000)
    m[k == 2] &= np.uint64(0xFFF)
    m[k == 3] = (np.uint64(1 << 52) - m[k == 3] % np.uint64(9)) & np.uint64((1 << 52) - 1)
    e = np.where(np.arange(n) % 3 == 0, rng.integers(0, 2047, n), rng.integers(990, 1060, n)).astype(np.uint64)
    s = rng.integers(0, 2, n, dtype=np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


@pytest.mark.parametrize("ulp", [-1.0, 0.0, 1.0])
def test_division_and_square_root(fp, ulp):
    fp.set_ulp(ulp)
    rng = np.random.default_rng(3)
    a, b = mantissas(rng, N), mantissas(rng, N)
    b2 = (a.view(np.uint64) + rng.integers(0, 5, N, dtype=np.uint64)).view(np.float64)  # quotients near 1
    sa, sb = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    with np.errstate(all="ignore"):
        for x, y in ((a, b), (a, b2), (a * b, b), (sa, sb), (np.ones(N), b)):
            assert same(fp(20, x, y), x / y)
        for x in (np.abs(a), SPECIAL, a, np.abs(b2) * np.abs(b2)):
            assert same(fp(21, x), np.sqrt(x))
    fp.set_ulp(0.0)


def test_rounding_and_comparison(fp):
    rng = np.random.default_rng(4)
    y = np.concatenate([rng.uniform(-5e5, 5e5, N), rng.uniform(-3, 3, N), np.arange(-4000, 4000) / 2.0, [0.0, -0.0]])
    y = np.concatenate([y, np.nextafter(y, 1e9), np.nextafter(y, -1e9)])
    y = y[np.abs(y) < 2.0 ** 19 - 1]
    assert same(fp(22, y), np.rint(y))
    k = np.concatenate([np.arange(-5000, 5000), rng.integers(-(1 << 20) + 1, 1 << 20, N)]).astype(np.float64)
    assert np.array_equal(fp(23, k), k)
    x = np.concatenate([mantissas(rng, N), SPECIAL])
    z = np.concatenate([mantissas(rng, N), SPECIAL[::-1]])
    with np.errstate(all="ignore"):
        assert same(fp(24, x), 0.5 * x)
    h = np.concatenate([rng.uniform(2.0 ** -11, 0.5, N), 2.0 ** -np.arange(2.0, 12.0), [np.nextafter(0.5, 0)],
                        np.rint(rng.uniform(1, 2, N) * 2.0 ** 40) * 2.0 ** rng.integers(-51, -41, N)])
    assert same(fp(28, h), 1.0 - h)
    ok = ~np.isnan(x) & ~np.isnan(z)
    assert np.array_equal(fp(25, x[ok], z[ok]), (x[ok] < z[ok]).astype(np.float64))


RANGES = {"exp": (-760, 720), "expm1": (-60, 720), "log": (1e-12, 1e3), "log1p": (-0.9, 30), "sin": (-2e4, 2e4),
          "cos": (-2e4, 2e4), "tanh": (-30, 30), "atan": (-50, 50), "asinh": (-40, 40)}


@pytest.mark.parametrize("fn", sorted(RANGES))
def test_functions_match_the_plain_build(fp, fn):
    rng = np.random.default_rng(5)
    lo, hi = RANGES[fn]
    x = np.concatenate([rng.uniform(lo, hi, N), rng.uniform(-1, 1, N) * 0.4, rng.uniform(-1, 1, N) * 2.0 ** rng.integers(-60, 8, N),
                        SPECIAL])
    if fn == "log":
        x = np.concatenate([np.abs(x), mantissas(rng, N)])
    if fn == "log1p":
        x = x[(x > -1.0) | np.isnan(x)]
    assert same(fp(O.DETMATH[fn], x), O.detmath(fn, x))


def test_two_argument_functions_match_the_plain_build(fp):
    rng = np.random.default_rng(6)
    sx, sy = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    x, y = np.concatenate([rng.uniform(-3, 3, N), sx]), np.concatenate([rng.uniform(-3, 3, N), sy])
    assert same(fp(8, x, y), O.detmath("atan2", x, y))
    b, e = np.exp(rng.uniform(-70, 30, N)), rng.uniform(-6, 6, N)
    assert same(fp(10, b, e), O.detmath("pow", b, e))
