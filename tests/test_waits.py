"""Calls whose name lacks "_async" return when their work is done: behind a long
queue on the context's stream the stream is empty after them, for lists that
go through the host ring and for longer ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _busy(pgb, a, torch):
    """Queue some tens of milliseconds of trial actions on the context's stream."""
    k = 400000
    b = torch.zeros((k, 2), dtype=torch.int32, device="cuda")
    x = torch.zeros((k, 3), dtype=torch.float64, device="cuda")
    out = torch.empty(k, dtype=torch.float64, device="cuda")
    work = torch.empty(2 * k, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):
        a._chk(a.lib.pgb_trial_actions_device_async(a.h, b.data_ptr(), x.data_ptr(), k, 1, pgb.PGB_ACTION_FULL, out.data_ptr(),
                                                    work.data_ptr()))
    return b, x, out, work


@pytest.mark.parametrize("k", [1, 40, 7000])
def test_updates_are_done_on_return(pgb, k):
    torch = pytest.importorskip("torch")
    n, m = 64, 128
    L = pgb.worldlines.box_side(n)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 1, extent=2 * n)
    a = pgb.Action(L, m, 2 * n, 0.004, 6.0596)
    a.load(cfg)
    stream = torch.cuda.ExternalStream(a.lib.pgb_stream(a.h))
    j = np.arange(k)
    beads = np.ascontiguousarray(np.stack([j % m, j // m], 1).astype(np.int32))
    pos = np.ascontiguousarray(cfg["pos"][beads[:, 0], beads[:, 1]])
    keep = _busy(pgb, a, torch)
    assert not stream.query()
    a.update_beads(beads, pos)
    assert stream.query()
    keep = _busy(pgb, a, torch)
    at = beads[:, 0], beads[:, 1]
    a.set_beads(beads, pos, cfg["next"][at], cfg["prev"][at], cfg["on"][at])
    assert stream.query()
    del keep
    a.plain_seed(3)
    a.plain_worm_run(1, mbar=16, temperature=1.0 / (m * 0.004), initial_num_particles=n, window=1, mu=0.0)
    assert stream.query()
