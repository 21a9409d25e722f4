"""Inputs and results in host memory: calls on both sides of every size limit
give the same values, many updates wrap the input ring before a wait, and
handles share pinned blocks without sharing data.  Equality is bitwise: the
kernels are the same."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _action(pgb, n=12, m=250, seed=1, action="gsf", precision=0):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, seed)
    a = pgb.Action(L, m, n, 0.004, 6.0596, action=action, precision=precision)
    a.load(cfg)
    return a, cfg, L


@pytest.mark.parametrize("precision", [0, 1])
def test_lists_beyond_the_direct_limit(pgb, precision):
    a, cfg, L = _action(pgb, precision=precision)
    rng = np.random.default_rng(3)
    beads = np.stack([rng.integers(0, 250, 2500), rng.integers(0, 12, 2500)], 1).astype(np.int32)
    pos = rng.uniform(-0.5 * L, 0.5 * L, (2500, 3))
    whole, _ = a.bead_actions(beads, mode=pgb.PGB_ACTION_BARE)
    tri = a.trial_actions(beads, pos, mode=pgb.PGB_ACTION_BARE)
    for i in range(0, 2500, 500):
        part, s = a.bead_actions(beads[i:i + 500], mode=pgb.PGB_ACTION_BARE)
        # FP64: other kernels from 1216 beads on, the same pairs in another order
        assert np.max(np.abs(part - whole[i:i + 500]) / np.maximum(np.abs(part), 1.0)) <= (0.0 if precision else 1e-12)
        assert s == pytest.approx(part.sum(), rel=1e-14)
        got = a.trial_actions(beads[i:i + 500], pos[i:i + 500], mode=pgb.PGB_ACTION_BARE)
        scale = np.maximum(1.0, np.maximum(np.abs(part), np.abs(got)))
        assert np.max(np.abs(got - tri[i:i + 500]) / scale) <= (0.0 if precision else 1e-12)


def test_updates_wrap_the_ring(pgb):
    a, cfg, L = _action(pgb)
    rng = np.random.default_rng(5)
    want = cfg["pos"].copy()
    for k in [1, 3000, 700, 5000] + [900] * 12:           # past the ring's half, and round it
        b = np.stack([rng.integers(0, 250, k), rng.integers(0, 12, k)], 1).astype(np.int32)
        _, first = np.unique(b[:, 0] * 12 + b[:, 1], return_index=True)
        b = np.ascontiguousarray(b[first])
        p = rng.uniform(-0.5 * L, 0.5 * L, (len(b), 3))
        a.update_beads(b, p)
        want[b[:, 0], b[:, 1]] = p
    assert np.array_equal(a.positions(), want)


def test_wave_vector_lists_on_both_sides(pgb):
    a, cfg, L = _action(pgb, n=20, m=32, precision=pgb.PGB_MIXED)
    q = (2 * np.pi / L) * np.random.default_rng(2).integers(-5, 6, (9000, 3))
    s, f = a.ssf(q), a.isf(q)                             # list and results too large
    for i in (0, 8000):
        assert np.array_equal(a.ssf(q[i:i + 100]), s[i:i + 100])
        assert np.array_equal(a.isf(q[i:i + 100]), f[i:i + 100])


def test_handles_in_threads_share_blocks_not_data(pgb):
    from pimc_gb300 import worldlines as wl
    from pimc_gb300.gp import GaussianProcess
    w = wl.workload_gp(points=200, num_ptcl=8, num_slices=25, seed=2)
    ref = GaussianProcess(w["training"], **w["params"])(w["pos"])
    acts = [_action(pgb, seed=s)[0].bead_actions([[5, 3], [6, 3]])[0] for s in range(4)]
    bad = []

    def work(s):
        for _ in range(10):
            g = GaussianProcess(w["training"], **w["params"])
            a = _action(pgb, seed=s)[0]
            if not (np.array_equal(g(w["pos"]), ref) and np.array_equal(a.bead_actions([[5, 3], [6, 3]])[0], acts[s])):
                bad.append(s)
            g.close()
            a.close()
    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
