"""The FP64 iterations of fp64_light.cuh (quotient and eighth root from an FP32
estimate) and its integer conversions, restated in numpy, against exact
results.  Estimates are taken at the worst error that the FP32 functions may
have (two ulp either way), so the bars hold for every implementation of them:
each iteration leaves less than 1e-20 of that, and its last FP64 operation
rounds once or twice, so two ulp (4.4e-16) bound the result."""
import numpy as np
import pytest

U = 2.0 ** -24
rng = np.random.default_rng(3)
X = np.concatenate([np.exp(rng.uniform(np.log(2.0 ** -99), np.log(2.0 ** 99), 200000)), [1.0, 2.0, 1e-24, 1.5, 4.0]])
BAR = 2 * 2.0 ** -52


def fma(a, b, c):
    """a b + c rounded once (through extended precision)."""
    return (np.asarray(a, np.longdouble) * b + c).astype(np.float64)


def seed(v, off):
    return (np.float32(v) * np.float32(1 + off)).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("off", [0.0, 2 * U, -2 * U])
def test_quotient(off):
    a, b = X, rng.permutation(X)
    r0 = seed(1.0 / b.astype(np.float32), off)
    r = fma(r0, fma(-b, r0, 1.0), r0)
    q = a * r
    y = fma(fma(-b, q, a), r, q)
    ref = np.asarray(a, np.longdouble) / b
    assert np.max(np.abs(y / ref - 1)) < BAR


@pytest.mark.parametrize("off", [0.0, 4 * U, -4 * U])
def test_eighth_root(off):
    y = seed(X.astype(np.float32).astype(np.float64) ** -0.125, off)
    y2 = y * y
    y4 = y2 * y2
    h = fma(-X, y4 * y4, 1.0)
    r = fma(y, h * fma(h, 0.0703125, 0.125), y)
    ref = np.asarray(X, np.longdouble) ** np.longdouble(-0.125)
    assert np.max(np.abs(r / ref - 1)) < BAR


def widen(x):
    b = x.view(np.uint32).astype(np.uint64)
    hi = (((b & 0x7fffffff) >> np.uint64(3)) + np.uint64(0x38000000)) | (b & np.uint64(0x80000000))
    return ((hi << np.uint64(32)) | ((b << np.uint64(29)) & np.uint64(0xffffffff))).view(np.float64)


def narrow(x):
    v = x.view(np.uint64)
    hi, lo = (v >> np.uint64(32)).astype(np.uint32), v.astype(np.uint32)
    with np.errstate(over="ignore"):
        l = lo + np.uint32(0x0fffffff) + ((lo >> np.uint32(29)) & np.uint32(1))
        h = (hi & np.uint32(0x7fffffff)) + (l < lo).astype(np.uint32)
        f = ((h << np.uint32(3)) | (l >> np.uint32(29))) - np.uint32(0xc0000000)
    return (f | (hi & np.uint32(0x80000000))).view(np.float32)


def test_conversions_are_exact():
    s = rng.choice([-1.0, 1.0], X.size)
    x = (X * s)
    ties = (x.astype(np.float32).astype(np.float64).view(np.uint64) & ~np.uint64(0x1fffffff) | np.uint64(0x10000000)).view(np.float64)
    for v in (x, ties):
        assert np.array_equal(narrow(v), v.astype(np.float32))
    f = x.astype(np.float32)
    assert np.array_equal(widen(f), f.astype(np.float64))
