"""The pipelined schedule against the grouped one: the same chains.

Draws are indexed by walker, step and move, and a move reads the configuration
its predecessor left however the work of a team is ordered, so the positions
and counters are equal.  Teams of one to sixteen warps, worldlines shorter
than a warp, bridges longer than one, Mbar = 2, odd and ragged particle
numbers, and bridges whose ends the move before has just moved (few particles).
"""
import numpy as np
import pytest

import pimc_gb300 as pgb

pytestmark = pytest.mark.gpu

N = [2, 3, 5, 9, 17, 31, 33, 60, 70, 63, 2, 3, 2, 9, 17]
M = [10, 12, 20, 34, 66, 40, 80, 62, 250, 244, 8, 30, 130, 36, 70]
MBAR = [4, 6, 8, 16, 32, 16, 32, 30, 40, 32, 2, 16, 64, 18, 40]
WIDE = ([127, 101, 64], [60, 90, 70], [32, 40, 64])


def _chains(n, m, mbar, schedule, steps=6):
    tau = 0.00400802
    m = np.array(m)
    w = pgb.Walkers(n, m, 1.0 / (tau * m), (np.array(n) / 0.02198) ** (1 / 3.0), mbar, tau, 6.0596, seed=7,
                    p_com=0.1, threads_per_walker=schedule)
    w.init()
    w.run(steps)
    st = w.stats()
    counts = [(s["attempted"], s["accepted"], s["bead_updates"]) for s in st]
    pos = [w.positions(i).copy() for i in range(len(n))]
    w.close()
    return counts, pos


@pytest.mark.parametrize("schedule", [5008, 5016, 6000, 6008, 6016])
def test_same_chains(schedule):
    for sizes in ((N, M, MBAR), WIDE) if schedule >= 6000 else ((N, M, MBAR),):
        want, at = _chains(*sizes, 8008)
        got, here = _chains(*sizes, schedule)
        assert got == want
        for a, b in zip(here, at):
            assert np.array_equal(a, b)
