"""g(r)'s counts where the FP32 bin is least certain: boxes whose first sides are
longer than the one that the bins are made of, and beads outside the box.
Counts are integers and have to be those of the FP64 binning, nR =
int(|r_j - r_i| / dSep) with the nearest image, so the normalised histograms
are equal bit for bit."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _histogram(pos, side):
    m, n, _ = pos.shape
    inv = 1.0 / side
    dsep = 0.5 * math.sqrt(3.0) * side[2] / 50.0
    i, j = np.triu_indices(n, 1)
    hist = np.zeros(50, dtype=np.int64)
    for s in range(m):
        d = pos[s, j] - pos[s, i]
        d = d - side * np.floor(d * inv + 0.5)
        r = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
        b = (r / dsep).astype(np.int64)
        hist += np.bincount(b[b < 50], minlength=50)[:50]
    g = np.zeros(50)
    for k in range(50):
        dv = math.pow((k + 1) * dsep, 3.0) - math.pow(k * dsep, 3.0)
        g[k] = 1.0 * (n - 1) / (1.0 * n) * (1.0 * hist[k] / float(hist.sum())) * (
            0.5 * (3.0 / (2.0 * math.pi) * (side[0] * side[1] * side[2])) / dv)
    return g


@pytest.mark.parametrize("ratio,spread", [(1.0, 1.0), (6.0, 1.0), (64.0, 1.0), (1000.0, 1.0), (1.0, 7.0)])
def test_counts(pgb, ratio, spread):
    n, m = 192, 40
    side = np.array([29.0, 28.0, 27.0 / ratio])
    rng = np.random.default_rng(int(ratio))
    cfg = pgb.worldlines.seeded_worldlines(n, m, 9.0, 6.0596, 0.004, 1)
    # a slice's beads about one place, so that pairs fall into the bins at all
    pos = rng.uniform(-0.5, 0.5, (m, 1, 3)) * side * spread + rng.uniform(-0.5, 0.5, (m, n, 3)) * side[2]
    cfg["pos"] = np.ascontiguousarray(pos if spread > 1.0 else pos - side * np.floor(pos / side + 0.5))
    a = pgb.Action(side, m, n, 0.004, 6.0596)
    a.load(cfg)
    assert np.array_equal(a.pair_correlation(-1), _histogram(cfg["pos"], side))


@pytest.mark.parametrize("n,m", [(32, 305), (33, 305), (2, 304)])
def test_counts_of_many_small_slices(pgb, n, m):
    side = np.array([9.0, 9.0, 9.0])
    cfg = pgb.worldlines.seeded_worldlines(n, m, 9.0, 6.0596, 0.004, 1)
    cfg["pos"] = np.random.default_rng(n).uniform(-4.5, 4.5, (m, n, 3))
    a = pgb.Action(side, m, n, 0.004, 6.0596)
    a.load(cfg)
    assert np.array_equal(a.pair_correlation(-1), _histogram(cfg["pos"], side))
