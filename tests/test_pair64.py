"""The FP64 bead actions' dispatch: one bead, clusters of CTAs, one warp a bead
and the trial forms, against the oracle's per-bead action.

Tolerance: every form sums the same pair terms (each within 2e-16 relative of
the oracle's), at most n^2 of them, in another order: 1e-12 of max(|U|, 1), as
for every FP64 action here.  A trial difference is held to the larger action.
"""
import numpy as np
import pytest

from helpers import make_pair, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(9, 8, 3), (33, 6, 31), (64, 6, 40), (65, 4, 160), (257, 4, 5), (40, 4, 911), (40, 4, 912), (40, 4, 1216),
         (70, 4, 2047), (70, 4, 2048)]


def _setup(pgb, oracle_lib, n, m, rc, worm, shift_box=0.0):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 31 + n)
    if worm:
        cfg = pgb.worldlines.open_worm(cfg, head=(1, n - 1), tail=(3, n - 1))
    cfg["pos"][0, 0] += shift_box * L                  # a bead stored outside the box
    return make_pair(pgb, oracle_lib, cfg, L, m, n, 0.004, 6.0596, rc=rc, action="gsf") + (cfg, L)


@pytest.mark.parametrize("n,m,k", SIZES)
@pytest.mark.parametrize("rc", [None, 5.0])
@pytest.mark.parametrize("worm", [False, True])
def test_forms_against_oracle(pgb, oracle_lib, n, m, k, rc, worm):
    a, o, cfg, L = _setup(pgb, oracle_lib, n, m, rc, worm)
    rng = np.random.default_rng(k)
    beads = np.stack([rng.integers(0, m, k), rng.integers(0, n, k)], 1).astype(np.int32)
    pos = rng.uniform(-0.5 * L, 0.5 * L, (k, 3))
    pos[0] = (0.5 * L, -0.5 * L, 0.0)                  # on the box edge
    some = np.unique(np.concatenate([[0, k - 1], rng.integers(0, k, 12)]))
    for shift, mode in ((1, 0), (2, 0), (1, 1), (1, 2)):
        o.set_shift(shift)
        got, _ = a.bead_actions(beads, shift=shift, mode=mode)
        tri = a.trial_actions(beads, pos, shift=shift, mode=mode)
        for i in some:
            s, p = (int(x) for x in beads[i])
            want = o.bead_action(s, p, mode)
            assert rel_err([got[i]], [want]) <= 1e-12, (shift, mode, i)
            old = cfg["pos"][s, p].copy()
            o.update_bead(s, p, pos[i])
            new = o.bead_action(s, p, mode) if cfg["on"][s, p] else 0.0
            o.update_bead(s, p, old)
            assert abs(tri[i] - (new - want)) <= 1e-12 * max(1.0, abs(new), abs(want)), (shift, mode, i)
    o.set_shift(1)


@pytest.mark.parametrize("shift_box", [1.0, -2.0, 40.0])
def test_beads_outside_the_box_take_the_direct_form(pgb, oracle_lib, shift_box):
    a, o, _, _ = _setup(pgb, oracle_lib, 20, 4, None, False, shift_box)
    beads = np.array([[0, 0], [0, 1], [0, 19], [1, 0]], np.int32)
    got, _ = a.bead_actions(beads)
    assert rel_err(got, [o.bead_action(int(s), int(p)) for s, p in beads]) <= 1e-12


@pytest.mark.parametrize("n,m", [(2, 4), (32, 6), (33, 6), (64, 6), (65, 8), (129, 6)])
@pytest.mark.parametrize("action", ["primitive", "gsf", "li_broughton"])
def test_slice_terms_row_blocks(pgb, oracle_lib, n, m, action):
    """Row blocks of 32 and 64 beads, several blocks a slice, the levels that
    the energy, the full action and the virial ask for (1e-11 for the virial's
    products of sums, as elsewhere), twice: the arrival counters return to 0."""
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 7 + n)
    if n > 8:
        cfg = pgb.worldlines.permute(cfg, [(1, 4), (2, 5, 7)])
    a, o = make_pair(pgb, oracle_lib, cfg, L, m, n, 0.004, 6.0596, action=action, mu=-3.0)
    for _ in range(2):
        assert rel_err(a.energy(), o.energy()) <= 1e-12
        assert rel_err(a.virial(), o.virial()) <= 1e-11
        assert abs(a.full_action() - o.full_action()) <= 1e-12 * max(1.0, abs(o.full_action()))
        assert abs(a.kinetic_action() - o.kinetic_action()) <= 1e-12 * max(1.0, abs(o.kinetic_action()))
    t = a.slice_terms()
    for s in range(m):
        assert abs(t["vint"][s] - o.V_slice(s)[1]) <= 1e-12 * max(1, abs(t["vint"][s]))
        assert abs(t["g2"][s] - o.slice_fn("gradVSquared_slice", s)) <= 1e-12 * max(1, t["g2"][s])
