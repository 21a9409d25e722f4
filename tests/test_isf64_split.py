"""FP64 F(q,tau) where its tau fill one CTA or several, with an odd number of
slices, for one vector and many, against NumPy in extended precision.

Tolerance: a density is within n 1e-13 (as for the densities' own tests), a
product of two within 2 n of that, the sum over m of them, over n m, within
2 n 1e-13, and its own roundings, m 2^-53 of at most n.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [5, 62, 253, 254, 256, 258, 511])
@pytest.mark.parametrize("nq", [1, 30])
def test_split_tau(pgb, m, nq):
    n = 6
    L = pgb.worldlines.box_side(n)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, m)
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    q = np.random.default_rng(nq).normal(0, 1.5, (nq, 3))
    ph = np.einsum("mnd,qd->qmn", cfg["pos"].astype(np.longdouble), q.astype(np.longdouble))
    re, im = np.cos(ph).sum(-1), np.sin(ph).sum(-1)
    F = np.stack([(re * np.roll(re, -k, 1) + im * np.roll(im, -k, 1)).sum(1) for k in range(m // 2 + 1)], 1) / (n * m)
    got = a.isf(q)
    assert got.shape == F.shape
    assert np.max(np.abs(got - F)) <= n * (2e-13 + m * 2.0 ** -53)
