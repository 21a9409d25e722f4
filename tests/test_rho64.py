"""FP64 densities: lattice vectors from tables of powers, mirrored lists, other
vectors, few and many vectors a slice, several chunks of beads, against NumPy
in extended precision phases.

Tolerance: a power of the tables carries at most 2 log2(n) + 2 roundings and a
product of three of them 20; with the phases' rounding (|q . r| <= 64 pi) a
term is within 1e-13, n terms within n 1e-13.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(L, rng):
    g = np.arange(-3, 4)
    full = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    lat = (2 * np.pi / L) * full
    some = (2 * np.pi / L) * rng.integers(-40, 41, (301, 3))
    other = rng.normal(0, 2.0, (37, 3))
    edge = (2 * np.pi / L) * np.array([[64, 0, -64], [65, 1, 0], [0, 0, 0], [1, 0, 0], [-1, 0, 0]])
    return dict(mirrored=lat, even=np.concatenate([lat[:171], lat[172:]]), scattered=some, other=other, edge=edge,
                mixed=np.concatenate([some[:40], other, lat[:60]]), one=some[:1], few=some[:33])


@pytest.mark.parametrize("n,m", [(7, 4), (64, 6), (200, 4)])
def test_densities(pgb, n, m):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n)
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    for name, q in _lists(L, np.random.default_rng(n)).items():
        ph = np.einsum("mnd,qd->qmn", cfg["pos"].astype(np.longdouble), q.astype(np.longdouble))
        want = np.stack([np.cos(ph).sum(-1), np.sin(ph).sum(-1)], -1).astype(np.float64)
        tol = n * 1e-13
        assert np.max(np.abs(a.rhoq(q) - want)) <= tol, name
        z = want[..., 0] + 1j * want[..., 1]
        F = np.stack([(z * np.conj(np.roll(z, -k, 1))).real.sum(1) for k in range(m // 2 + 1)], 1) / (n * m)
        # |rho| <= n: a product of two densities is within 2 n tol, F within 2 tol and its own sums
        assert np.max(np.abs(a.isf(q) - F)) <= 3 * tol, name
        assert np.max(np.abs(a.ssf(q) - F[:, 0])) <= 3 * tol, name
        inside = cfg["pos"][..., 0] ** 2 + cfg["pos"][..., 1] ** 2 < 9.0
        zc = ((np.cos(ph) * inside[None]).sum(-1) ** 2 + (np.sin(ph) * inside[None]).sum(-1) ** 2).sum(1) / m
        assert np.max(np.abs(a.ssf_cylinder(q, 3.0)[0] - zc.astype(np.float64))) <= 3 * n * tol, name
