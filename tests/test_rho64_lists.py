"""FP64 densities on both sides of the rules that choose their form: lists of
few vectors, short paths, vectors off the lattice among few and many lattice
ones, mirrored lists, the cylinder's mask, one to eight CTAs a slice.

Tolerance: a term's phase q . r is off by at most three roundings of its
components and two of their sum, its sine and cosine by an ulp; n terms and
their sum of at most n add n / 2 ulps of n.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def exact(pos, q):
    ph = np.einsum("mnd,qd->qmn", pos.astype(np.longdouble), q.astype(np.longdouble))
    return ph, np.stack([np.cos(ph).sum(-1), np.sin(ph).sum(-1)], -1)


def bound(pos, q):
    phase = np.abs(pos)[None].max((1, 2)) @ np.abs(q).T       # (1, nq): |q| . |r| at most
    n = pos.shape[1]
    return (n * EPS * (5 * phase[0] + 4 + n))[:, None, None]


def _lists(L, rng):
    lat = (2 * np.pi / L) * rng.integers(-9, 10, (80, 3))
    other = rng.normal(0, 2.0, (80, 3))
    g = (2 * np.pi / L) * np.stack(np.meshgrid(*[np.arange(-2, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return dict(one=lat[:1], off=other[:1], few=lat[:23], few_off=other[:24], rule=np.concatenate([lat[:30], other[:4]]),
                mixed=np.concatenate([other[:70], lat, -lat[:20]]), others=other, grid=g, far=np.concatenate([lat[:40] * 60, other[:3] * 1e9]))


@pytest.mark.parametrize("n,m", [(5, 30), (9, 33), (33, 31), (40, 60), (26, 100), (130, 34)])
def test_lists(pgb, n, m):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n)
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    inside = cfg["pos"][..., 0] ** 2 + cfg["pos"][..., 1] ** 2 < 9.0
    for name, q in _lists(L, np.random.default_rng(n)).items():
        q = np.ascontiguousarray(q)
        ph, want = exact(cfg["pos"], q)
        tol = bound(cfg["pos"], q)
        assert np.all(np.abs(a.rhoq(q) - want) <= tol), name
        if name == "far":
            continue
        z = ((np.cos(ph) * inside).sum(-1) ** 2 + (np.sin(ph) * inside).sum(-1) ** 2).sum(1) / m
        assert np.all(np.abs(a.ssf_cylinder(q, 3.0)[0] - z) <= 3 * n * tol[:, 0, 0]), name


@pytest.mark.parametrize("n,m,nq", [(5, 8, 4609), (9, 31, 1200), (24, 24, 1500), (40, 31, 1663)])
def test_many_vectors_of_short_paths(pgb, n, m, nq):
    """Both forms of a short path: many vectors on the lattice, a few off it."""
    L = 2.9 * n ** (1.0 / 3.0)
    rng = np.random.default_rng(nq)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n)
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    q = (2 * np.pi / L) * rng.integers(-9, 10, (nq, 3))
    q[::97] = rng.normal(0, 2.0, (len(q[::97]), 3))
    for part in (q, q[:400]):
        part = np.ascontiguousarray(part)
        assert np.all(np.abs(a.rhoq(part) - exact(cfg["pos"], part)[1]) <= bound(cfg["pos"], part))
