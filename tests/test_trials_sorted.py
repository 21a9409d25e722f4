"""Trials sorted by bead against the same trials one by one: the same bits, for
every parity and mode, repeated and rare beads, groups of every size, inactive
beads, an open worm, and output buffers that rule sorting out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(pgb, a, beads, pos, shift, mode, offset):
    import torch
    k = len(beads)
    d_b, d_p = torch.from_numpy(beads).cuda(), torch.from_numpy(pos).cuda()
    out = torch.zeros(k, dtype=torch.float64, device="cuda")
    work = torch.zeros(2 * k + 1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    a._chk(a.lib.pgb_trial_actions_device_async(a.h, d_b.data_ptr(), d_p.data_ptr(), k, shift, mode, out.data_ptr(),
                                                work.data_ptr() + 8 * offset))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("n,m,k", [(300, 4, 9000), (257, 3, 9730), (64, 8, 40000)])
@pytest.mark.parametrize("action", ["primitive", "gsf", "li_broughton"])
def test_sorted_trials_have_the_unsorted_bits(pgb, n, m, k, action):
    L = 2.9 * n ** (1.0 / 3.0)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, n)
    cfg = pgb.worldlines.open_worm(cfg, head=(0, n - 1), tail=(2, n - 1))
    a = pgb.Action(L, m, n, 0.004, 6.0596, action=action, precision=pgb.PGB_MIXED)
    a.load(cfg)
    rng = np.random.default_rng(k)
    p = np.minimum(rng.geometric(4.0 / n, k) - 1, n - 1)              # few beads often, many rarely
    beads = np.stack([rng.integers(0, m, k), p], 1).astype(np.int32)
    beads[:3] = [[1, n - 1], [-1, 0], [0, n]]                         # switched off, outside
    pos = rng.uniform(-0.5 * L, 0.5 * L, (k, 3))
    for shift, mode in ((1, 0), (2, 0), (1, 1), (1, 2)):
        got = _call(pgb, a, beads, pos, shift, mode, 0)
        # a work buffer off a 16-byte boundary leaves no room for the sorted records
        assert np.array_equal(got, _call(pgb, a, beads, pos, shift, mode, 1)), (shift, mode)
        one = np.concatenate([a.trial_actions(beads[i:i + 500], pos[i:i + 500], shift=shift, mode=mode)
                              for i in range(3, k - 500, k // 5)])
        idx = np.concatenate([np.arange(i, i + 500) for i in range(3, k - 500, k // 5)])
        assert np.array_equal(got[idx], one), (shift, mode)
        assert np.all(got[:3] == 0.0)
        assert np.array_equal(a.trial_actions(beads[3:], pos[3:], shift=shift, mode=mode), got[3:])
