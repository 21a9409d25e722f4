"""The walkers' chains, pinned.

A walker's moves draw from its own stream and decide by FP32 pair sums, so a
change of the walks, the tests of a run, the removal of a run's beads, the
deviates or the split of a sum over warps either leaves the chain as it was or
shows in the first sweeps.  The figures (moves attempted and accepted, beads
moved, closed steps, errors, and a checksum of the positions, links and bead
counts) are those of the form that walks bead by bead, tests and removes one
bead after another and draws one attempt a lane.  The sizes cover worldlines
shorter than a warp and not a multiple of it, Mbar from 2 to 64, one bead a
slice, the edges between the walkers' schedules, open and closed ensembles and
both diagonal moves.
"""
import zlib

import numpy as np
import pytest

import pimc_gb300 as pgb

pytestmark = pytest.mark.gpu

SMALL = ([1, 2, 3, 5, 17, 31], [4, 6, 10, 30, 34, 66], [2, 4, 8, 16, 32, 64])
LARGE = ([32, 33, 63, 64, 65, 130], [30, 32, 34, 62, 96, 128], [16, 8, 32, 60, 64, 32])


@pytest.mark.parametrize("sizes,window,mu,diagonal,expected", [
    (SMALL, -1, 4.0, 0, (11623, 4862, 78432, 65, 0, 3424254923)),
    (LARGE, 1, -2.0, 0, (18323, 5829, 234375, 44, 0, 1156767131)),
    (SMALL, 1, -2.0, 1, (11656, 4885, 81494, 68, 0, 898956799)),
    (LARGE, -1, -20.0, 1, (18258, 7465, 297836, 26, 0, 4081702068)),
])
def test_chain(sizes, window, mu, diagonal, expected):
    n, m, mbar = sizes
    side = [(v / 0.02198) ** (1 / 3) for v in n]
    w = pgb.WormWalkers(n, m, side, mbar, 0.004, 6.0596, window=window, mu=mu, seed=11, diagonal_move=diagonal)
    w.seed_device(3)
    w.equilibrate(8)
    w.run(12)
    st = w.stats()
    image = np.zeros(w.state_bytes(), np.uint8)
    w.get_state(image)
    beads, slices = int((w.m.astype(np.int64) * w.capacity).sum()), int(w.m.sum())
    paths = zlib.crc32(image[: 24 * beads + 4 * slices].tobytes())
    w.close()
    assert (int(st["attempted"].sum()), int(st["accepted"].sum()), int(st["bead_updates"].sum()),
            int(st["samples"].sum()), int(st["error"].sum()), paths) == expected
