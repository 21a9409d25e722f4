"""Permutation cycles, winding and g(r) at the edges of their kernels: slices
that are not whole segments, several CTAs of beads, links that skip slices,
against walks and sums in NumPy (integer results equal; FP64 sums of at most
M N terms within 1e-12) and the oracle's histogram."""
import numpy as np
import pytest

from helpers import make_pair

pytestmark = pytest.mark.gpu


def _cycles(nxt, n, m):
    out = np.zeros(40)
    for i in range(n):
        s, p, wl, small = 0, i, 0, True
        while True:
            wl += 1
            small = small and not (s == 0 and p < i)
            s, p = (int(x) for x in nxt[s, p])
            if s == 0 and p == i:
                break
        if small and 0 < wl // m <= 40:
            out[wl // m - 1] += 1.0 * (wl // m) * (1.0 / n)     # the estimator's own products
    return out


@pytest.mark.parametrize("n,m", [(1, 2), (3, 1), (24, 15), (24, 16), (24, 17), (257, 34), (600, 6)])
def test_cycles_and_winding(pgb, n, m):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n + m)
    rng = np.random.default_rng(n)
    for s in range(0, m, 5):                              # exchanges on several slices
        perm = rng.permutation(n)
        cfg["next"][s, :, 1] = perm
        t = (s + 1) % m
        cfg["prev"][t, perm, 0], cfg["prev"][t, perm, 1] = s, np.arange(n)
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    nx = cfg["next"]
    W = cfg["pos"][nx[..., 0], nx[..., 1]] - cfg["pos"]
    W = (W - L * np.floor(W / L + 0.5)).sum((0, 1))
    for _ in range(2):                                    # the arrival counters return to 0
        assert np.array_equal(a.permutation_cycles(), _cycles(nx, n, m))
        sf = a.superfluid()
        assert np.max(np.abs(sf[1:4] - (W / L) ** 2)) <= 1e-12 * n * m


def test_cycles_through_links_that_skip_a_slice(pgb):
    n, m, L = 5, 18, 9.0
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 3)
    cfg["next"][4, 2] = (6, 2)                            # particle 2 skips slice 5
    a = pgb.Action(L, m, n, 0.004, 6.0596)
    a.load(cfg)
    want = np.zeros(40)
    for _ in range(n - 1):                                # 17 beads are not a whole cycle
        want[0] += 1.0 * (1.0 / n)
    assert np.array_equal(a.permutation_cycles(), want)


@pytest.mark.parametrize("n", [2, 33, 257])
def test_pair_histogram(pgb, oracle_lib, n):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, 6, L, 6.0596, 0.004, n)
    cfg["pos"][0, 1] = cfg["pos"][0, 0]                   # a pair at distance 0
    a, o = make_pair(pgb, oracle_lib, cfg, L, 6, n, 0.004, 6.0596)
    assert np.array_equal(a.pair_correlation(-1), o.pair_correlation(-1))
    assert np.array_equal(a.pair_correlation(0), o.pair_correlation(0))
