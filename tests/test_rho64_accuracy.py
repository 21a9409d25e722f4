"""The FP64 densities and F(q,tau) are as near to extended precision as the
plain form, a sine and a cosine of q . r a term, is in NumPy: a table must not
shift the phases (F(q,tau) averages out what differs from term to term, not
what all terms share).

Bound: one and a half times the plain form's own error, which is the rounding of its
phases and sums, and half an ulp of the result.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def correlation(re, im, m, n):
    return np.stack([(re * np.roll(re, -k, 1) + im * np.roll(im, -k, 1)).sum(1) for k in range(m // 2 + 1)], 1) / (n * m)


@pytest.mark.parametrize("n,m,qmax", [(9, 62, 2.0), (40, 62, 4.0), (100, 40, 3.0)])
def test_errors(pgb, n, m, qmax):
    L = pgb.worldlines.box_side(n)
    rng = np.random.default_rng(n)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n)
    cfg["pos"] = rng.uniform(-0.5 * L, 0.5 * L, (m, n, 3))
    top = int(qmax * L / (2 * np.pi))
    q = 2 * np.pi * rng.integers(-top, top + 1, (80, 3)) / L
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    ph = np.einsum("mnd,qd->qmn", cfg["pos"].astype(np.longdouble), q.astype(np.longdouble))
    re, im = np.cos(ph).sum(-1), np.sin(ph).sum(-1)
    ph = np.einsum("mnd,qd->qmn", cfg["pos"], q)
    plain = np.cos(ph).sum(-1), np.sin(ph).sum(-1)
    err = lambda x, y: float(np.linalg.norm((x - y).astype(np.float64)) / np.linalg.norm(y.astype(np.float64)))
    got = a.rhoq(q)
    want = np.stack([re, im], -1)
    assert err(got, want) <= 1.5 * err(np.stack(plain, -1), want) + 2.0 ** -54
    F = correlation(re, im, m, n)
    assert err(a.isf(q), F) <= 1.5 * err(correlation(*plain, m, n), F) + 2.0 ** -54
