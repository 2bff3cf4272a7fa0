"""The tridiagonal solvers' hypot (csrc/hypot.hpp), host side: below one ulp over the whole
range of doubles, unchanged by powers of two, and the results of C's hypot for zeros,
infinities and numbers next to overflow and underflow."""
import ctypes

import numpy as np
import pytest

import native


def _hypot(a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    out = np.empty_like(a)
    native.load().nc_hypot(ctypes.c_longlong(a.size), native.ptr(a), native.ptr(b), native.ptr(out))
    return out


def _pairs(seed, n=200000):
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(0.5, 1.0, n), rng.uniform(0.5, 1.0, n)
    return a, b * 2.0 ** -rng.integers(0, 60, n), rng


@pytest.mark.parametrize("seed", range(5))
def test_below_one_ulp(seed):
    a, b, rng = _pairs(seed)
    h = _hypot(a, b)
    exact = np.sqrt(np.longdouble(a) ** 2 + np.longdouble(b) ** 2)   # 64 bits of mantissa
    assert np.max(np.abs(np.longdouble(h) - exact) / np.spacing(h)) < 1.0
    assert np.array_equal(h, _hypot(b, a)) and np.array_equal(h, _hypot(-a, b))


@pytest.mark.parametrize("k", [-1000, -600, -461, -302, -300, -298, 298, 301, 600, 1020])
def test_unchanged_by_a_power_of_two(k):
    a, b, _ = _pairs(7)
    ok = (b * 2.0 ** max(k, -1000) != 0) & (np.ldexp(np.ldexp(b, k), -k) == b)   # exact in the target range
    assert ok.any()
    assert np.array_equal(_hypot(np.ldexp(a, k), np.ldexp(b, k))[ok], np.ldexp(_hypot(a, b), k)[ok])


def test_edges():
    big, tiny, inf = np.finfo(np.float64).max, 5e-324, np.inf
    cases = [(0, 0, 0), (0, 3, 3), (-4, 0, 4), (3, 4, 5), (3e-320, 4e-320, None), (tiny, tiny, None), (tiny, 0, tiny),
             (big, 0, big), (big, big, inf), (big, 1, big), (0.6 * big, 0.7 * big, None), (inf, 1, inf), (-inf, inf, inf),
             (1, 2.0 ** -53, 1), (1, 1e-300, 1), (1e-300, 1e300, 1e300)]
    a, b = np.array([c[0] for c in cases], float), np.array([c[1] for c in cases], float)
    got = _hypot(a, b)
    for x, y, g, (_, _, w) in zip(a, b, got, cases):
        if w is None:
            w = float(np.sqrt(np.longdouble(x) ** 2 + np.longdouble(y) ** 2))
            assert abs(g - w) <= np.spacing(w), (x, y)
        else:
            assert g == w, (x, y)
    assert np.all(np.isnan(_hypot(np.array([np.nan, 1, 0]), np.array([1, np.nan, np.nan]))))
