"""The FP64 Gaussian-process form's own root, third, exponential and reciprocal
root against extended precision, over their ranges: the ends where the library's
functions take over, the edges of the exponential's table intervals, arguments
around the powers of two, squares and cubes.

Bounds: as derived beside the functions, with 2^-9 ulp for the comparison
itself where the extended type has 64 bits.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(pgb, x, what):
    x = np.ascontiguousarray(x, dtype=np.float64)
    out = np.empty_like(x)
    lib = pgb._lib.load()
    dp = C.POINTER(C.c_double)
    assert lib.pgb_gp_math_check(x.ctypes.data_as(dp), len(x), what, out.ctypes.data_as(dp)) == 0
    return out


def _ulps(got, want):
    """The distance in ulps of the rounded exact value."""
    return np.abs((got.astype(np.longdouble) - want) / np.spacing(want.astype(np.float64)).astype(np.longdouble)).astype(float)


def _positive(rng, lo, hi, count=20000):
    x = np.exp2(rng.uniform(lo, hi, count))
    e = np.exp2(np.arange(int(lo) + 1, int(hi)).astype(float))
    near = np.concatenate([np.nextafter(e, 0), e, np.nextafter(e, np.inf)])
    squares = rng.integers(1, 1 << 26, 5000).astype(float) ** 2
    return np.concatenate([x, near, squares, np.nextafter(squares, np.inf)])


def test_roots(pgb):
    x = _positive(np.random.default_rng(1), -960, 960)
    assert np.max(_ulps(_run(pgb, x, 0), np.sqrt(x.astype(np.longdouble)))) <= 0.5 + 2.0 ** -9
    want = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.max(np.abs(_run(pgb, x, 3).astype(np.longdouble) / want - 1).astype(float)) <= 2.0 ** -52


def test_third(pgb):
    x = _positive(np.random.default_rng(2), -900, 1000)
    x = np.concatenate([x, 3.0 * np.arange(1.0, 4000.0), np.nextafter(3.0 * np.arange(1.0, 4000.0), 0), [0.0]])
    assert np.array_equal(_run(pgb, x, 1), x / 3.0)


def test_exponential(pgb):
    rng = np.random.default_rng(3)
    step = np.log(2.0) / 64
    edges = (np.arange(0, 64600) + 0.5) * step
    x = np.concatenate([rng.uniform(0, 40, 60000), rng.uniform(0, 700, 20000), np.exp2(rng.uniform(-60, 0, 5000)), edges[edges < 700],
                        np.nextafter(edges[edges < 700], 0), np.arange(0, 64000) * step, [0.0, np.nextafter(700.0, 0)]])
    x = x[x < 700]
    assert np.max(_ulps(_run(pgb, x, 2), np.exp(-x.astype(np.longdouble)))) <= 1.01 + 2.0 ** -9
    # from 700 on the library's function, which may leave the normal range
    y = np.array([700.0, 708.3, 720.0, 745.0, 746.0, 1e9, np.inf, np.nan])
    assert np.allclose(_run(pgb, y, 2), np.exp(-y), rtol=1e-15, atol=5e-324, equal_nan=True)
