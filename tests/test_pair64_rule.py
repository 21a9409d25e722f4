"""FP64 bead and trial actions on both sides of the rule that takes long lists
with a gradient term to the many-bead form: the same beads in one list and in
parts too short for it.  Two summation orders of the same pairs: within 1e-12 of
the actions' scale, as the forms are held to against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,k", [(40, 4, 624), (40, 4, 625), (64, 200, 799), (64, 200, 800), (200, 60, 193), (200, 60, 192),
                                   (16, 400, 1600), (16, 600, 2048)])
@pytest.mark.parametrize("action", ["gsf", "li_broughton"])
def test_one_list_and_parts(pgb, n, m, k, action):
    L = pgb.worldlines.box_side(n)
    rng = np.random.default_rng(k)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 1)
    g = int(np.ceil(n ** (1 / 3)))
    site = np.stack(np.unravel_index(rng.permutation(g ** 3)[:n], (g, g, g)), 1)
    r = (site + 0.5 + rng.uniform(-0.1, 0.1, (n, 3))) * (L / g) - 0.5 * L
    cfg["pos"] = np.ascontiguousarray(r[None] + rng.normal(0, 0.1, (m, n, 3)))
    a = pgb.Action(L, m, n, 0.004, 6.0596, action=action)
    a.load(cfg)
    beads = np.stack([rng.integers(0, m, k), rng.integers(0, n, k)], 1).astype(np.int32)
    pos = cfg["pos"][beads[:, 0], beads[:, 1]] + rng.normal(0, 0.1, (k, 3))
    whole, tri = a.bead_actions(beads)[0], a.trial_actions(beads, pos)
    for i in range(0, k, 90):
        part = a.bead_actions(beads[i:i + 90])[0]
        scale = np.maximum(1.0, np.abs(part).max())
        assert np.max(np.abs(part - whole[i:i + 90])) <= 1e-12 * scale
        assert np.max(np.abs(a.trial_actions(beads[i:i + 90], pos[i:i + 90]) - tri[i:i + 90])) <= 2e-12 * scale
