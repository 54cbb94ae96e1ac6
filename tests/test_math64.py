"""The FP64 functions of hxg_math64.cuh over their stated ranges and at the ends of
them, against numpy's extended precision (64-bit mantissa; its own error is below
0.01 ulp of FP64).  Bounds are those stated and derived beside each function, in
ulp of the exact result or in u = 2^-53."""
import ctypes as C
import os
import shutil
import subprocess
from fractions import Fraction as F

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hammurabix_b200", "csrc")
L = np.longdouble
PI = L("3.14159265358979323846264338327950288")
U = 2.0 ** -53
EXP, EXP_IN, RSQRT, SQRT, RCP, SINCOS, POW, SQRT_POS, DOT2 = range(9)


@pytest.fixture(scope="module")
def fn(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("math64") / "probe.so")
    subprocess.run([nvcc, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC,
                    "-o", so, os.path.join(HERE, "math64_probe.cu")], check=True)
    lib = C.CDLL(so)

    def call(f, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        t = [torch.from_numpy(v).cuda() for v in (a, a if b is None else np.ascontiguousarray(b))]
        o = [torch.zeros_like(t[0]) for _ in range(2)]
        p = [C.c_void_p(v.data_ptr()) for v in (*t, *o)]
        torch.cuda.synchronize()
        assert lib.probe(f, len(a), *p) == 0
        return [v.cpu().numpy() for v in o]
    return call


def _ulps(got, exact):
    """|got - exact| in ulp of exact."""
    u = np.spacing(np.abs(exact).astype(np.float64)).astype(L)
    return np.abs(got.astype(L) - exact) / u


def _rng():
    return np.random.Generator(np.random.PCG64(12))


def _wide(n=200000):
    """Positive normal numbers over most of the exponent range."""
    r = _rng()
    return np.ldexp(1 + r.random(n), r.integers(-950, 950, n))


@pytest.mark.parametrize("f", [EXP, EXP_IN])
def test_exp64(fn, f):
    r = _rng()
    a = np.concatenate([r.uniform(-681.99, 681.99, 400000), r.uniform(-1, 1, 100000),
                        r.uniform(-1e-3, 1e-3, 1000), np.ldexp(1.0, np.arange(-60, 10)),
                        [0.0, -0.0, 681.9, -681.9, 5e-324, -5e-324],
                        (np.arange(-2000, 2000) + 0.5) * (np.log(2.0) / 64)])
    got = fn(f, a)[0]
    assert _ulps(got, np.exp(a.astype(L))).max() <= 1.4
    assert got[np.flatnonzero(a == 0)].tolist() == [1.0, 1.0]


def test_exp64_outside_its_range(fn):
    a = np.array([682.0, 700.0, 709.7, 710.0, 1e300, np.inf, -682.0, -700.0, -740.0, -746.0, -1e300,
                  -np.inf, np.nan])
    got = fn(EXP, a)[0]
    with np.errstate(over="ignore", under="ignore"):
        want = np.exp(a.astype(L)).astype(np.float64)
    ok = np.isfinite(want) & (want > 1e-300)
    assert (np.abs(got - want)[ok] <= 4 * U * want[ok]).all()
    assert np.isnan(got[-1]) and np.isinf(got[3:6]).all() and (got[9:12] == 0).all()
    assert abs(got[8] - want[8]) <= 5e-324


def test_rsqrt64_and_sqrt64(fn):
    t = np.concatenate([_wide(), 1 + np.ldexp(_rng().random(1000), -40),
                        np.ldexp(1.0, np.arange(-1021, 1023)), [2.2250738585072014e-308, 1.7e308]])
    root = np.sqrt(t.astype(L))
    assert _ulps(fn(RSQRT, t)[0], 1 / root).max() <= 1.05
    got, inv = fn(SQRT, t)
    assert _ulps(got, root).max() <= 0.51
    assert _ulps(inv, 1 / root).max() <= 1.05


def test_rcp64(fn):
    d = np.concatenate([_wide(), -_wide(1000), np.ldexp(1.0, np.arange(-1021, 1021)),
                        1 + np.ldexp(_rng().random(1000), -45)])
    got = fn(RCP, d)[0]
    assert _ulps(got, 1 / d.astype(L)).max() <= 0.55
    p = np.ldexp(1.0, np.arange(-1000, 1000))
    assert (fn(RCP, p)[0] == 1 / p).all()       # the logistic step's 1 / (1 + 0)


def test_sqrt_pos(fn):
    v = np.concatenate([_wide(1000), [0.0, 5e-324, 1e-310, 1e-291, 1e-290, 1.1e-290]])
    assert _ulps(fn(SQRT_POS, v)[0], np.sqrt(v.astype(L)))[v > 0].max() <= 0.51
    assert fn(SQRT_POS, [0.0])[0][0] == 0


def test_sincos_quarter(fn):
    r = _rng()
    h = np.concatenate([r.uniform(-1, 1, 200000), r.uniform(-1e4, 1e4, 200000),
                        r.uniform(-2.0 ** 49, 2.0 ** 49, 20000), np.arange(-64, 65) / 2,
                        [2.0 ** 49 - 1, 1 - 2.0 ** 49, 1e-300, -1e-300, 0.0],
                        np.ldexp(1.0, np.arange(-60, 0))])
    s, c = fn(SINCOS, h)
    n = np.rint(h)
    f = ((h - n).astype(L)) * (PI / 2)          # exact difference
    a, b, k = np.sin(f), np.cos(f), n.astype(np.int64) & 3
    es = np.choose(k, [a, b, -a, -b])
    ec = np.choose(k, [b, -a, -b, a])
    assert np.abs(s - es).max() <= 2 * U and np.abs(c - ec).max() <= 2 * U
    for got, want, poly in ((s, es, (k & 1) == 0), (c, ec, (k & 1) == 1)):
        at = poly & (want != 0)
        assert (np.abs(got - want)[at] <= 2.4 * U * np.abs(want)[at]).all()
        assert (got[poly & (want == 0)] == 0).all()


def test_sincos_quarter_outside_its_range(fn):
    h = np.array([2.0 ** 49, 2.0 ** 49 + 0.5, -2.0 ** 50 - 1, 2.0 ** 60, 3e22, np.inf, np.nan])
    s, c = fn(SINCOS, h)
    fin = np.isfinite(h)
    k = np.mod(h[fin], 4.0)                     # exact
    assert (np.abs(s[fin] - np.sin(k.astype(L) * PI / 2)) <= 4 * U).all()
    assert (np.abs(c[fin] - np.cos(k.astype(L) * PI / 2)) <= 4 * U).all()
    assert np.isnan(s[~fin]).all() and np.isnan(c[~fin]).all()


@pytest.mark.parametrize("a", [-11.0 / 3.0, 6.0, -1.7, 0.4, 0.0, 1.0, -30.0])
def test_pow_k(fn, a):
    r = _rng()
    x = np.concatenate([np.exp(r.uniform(-12, 12, 200000)), np.ldexp(1.0, np.arange(-20, 20)),
                        1 + np.ldexp(r.uniform(-1, 1, 1000), -20), [0.7071, 1.4142, 0.70710678]])
    want = np.exp2(a * np.log2(x.astype(L)))
    # the oracle's own exponent carries 2^-64 of up to |a| 17.4 binary places
    tol = (1.5 * abs(a) + 4) * U + abs(a) * 17.4 * 2.0 ** -63
    assert (np.abs(fn(POW, x, np.full_like(x, a))[0] - want) <= tol * want).all()


def test_pow_k_outside_its_range(fn):
    x = np.array([0.0, 1e-320, 1e300, np.inf, np.nan, -1.0, 1e-200])
    a = np.array([2.0, 0.5, 5.0, 1.0, 1.0, 2.0, -8.0])
    got = fn(POW, x, a)[0]
    with np.errstate(all="ignore"):
        want = np.power(x, a)
    assert np.isnan(got[4]) and np.allclose(np.delete(got, 4), np.delete(want, 4), rtol=1e-14,
                                            atol=0)


def test_dot2_64(fn):
    """a b + c d of pairs from both ends of the arrays, exact in rationals."""
    r = _rng()
    a, b = r.uniform(-1, 1, 3000), r.uniform(-1, 1, 3000) * 2.5e22
    a[:500], b[:500] = np.cos(r.uniform(0, 6.3, 500)), -2.561e22
    hi, lo = fn(DOT2, a, b)
    for k in range(len(a)):
        x, y = F(a[k]) * F(b[k]), F(a[-1 - k]) * F(b[-1 - k])
        assert abs(F(hi[k]) + F(lo[k]) - (x + y)) <= F(4 * U * U) * (abs(x) + abs(y)), k
