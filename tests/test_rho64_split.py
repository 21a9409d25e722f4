"""FP64 densities with a slice's beads shared out: over the CTAs of a cluster
(few slices, more slices than fit at once, bead numbers that do not divide),
over the threads of a CTA (few vectors), and more vectors than one CTA takes,
against NumPy in extended precision.

Tolerance: as for the densities of one CTA, a term within 1e-13, n terms
within n 1e-13; adding the parts in another order stays inside it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(31, 4), (33, 40), (65, 10), (67, 156), (129, 4)])
@pytest.mark.parametrize("nq", [1, 33, 129, 700])
def test_split_densities(pgb, n, m, nq):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n)
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    rng = np.random.default_rng(nq)
    q = (2 * np.pi / L) * rng.integers(-9, 10, (nq, 3))
    if nq > 1:
        q[nq // 2:] = -q[: nq - nq // 2][::-1]                            # half of it mirrored
        q[0] = rng.normal(0, 2.0, 3)                                      # and one not on the lattice
    ph = np.einsum("mnd,qd->qmn", cfg["pos"].astype(np.longdouble), q.astype(np.longdouble))
    want = np.stack([np.cos(ph).sum(-1), np.sin(ph).sum(-1)], -1).astype(np.float64)
    assert np.max(np.abs(a.rhoq(q) - want)) <= n * 1e-13
