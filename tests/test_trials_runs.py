"""Trials of few beads: a bead's trials in several runs, which start anywhere in
the sorted list (one bead, one worldline, two beads whose runs meet, counts at
the run's length), against the unsorted form, bit for bit."""
import numpy as np
import pytest

from test_trials_sorted import _call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", ["bead", "worldline", "two", "edges"])
@pytest.mark.parametrize("action", ["primitive", "gsf"])
def test_runs(pgb, spread, action):
    n, m, k = 65, 6, 40000
    L = pgb.worldlines.box_side(n)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 1)
    a = pgb.Action(L, m, n, 0.004, 6.0596, action=action, precision=pgb.PGB_MIXED)
    a.load(cfg)
    rng = np.random.default_rng(4)
    i = np.arange(k)
    if spread == "bead":
        beads = np.stack([0 * i + 3, 0 * i + 7], 1)
    elif spread == "worldline":
        beads = np.stack([i % m, 0 * i + 64], 1)
    elif spread == "two":
        beads = np.stack([0 * i + 2, np.where(i < 1000, 1, 2)], 1)
    else:                                # 1, 63, 64, 65, 127, 128, 129 trials a bead, the rest on one
        c = np.array([1, 63, 64, 65, 127, 128, 129])
        p = np.concatenate([np.repeat(np.arange(7), c), np.full(k - c.sum(), 50)])
        beads = np.stack([0 * i + 5, p], 1)[rng.permutation(k)]
    beads = np.ascontiguousarray(beads.astype(np.int32))
    pos = rng.uniform(-0.5 * L, 0.5 * L, (k, 3))
    got = _call(pgb, a, beads, pos, 1, 0, 0)
    assert np.array_equal(got, _call(pgb, a, beads, pos, 1, 0, 1))
