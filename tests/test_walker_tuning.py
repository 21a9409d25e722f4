"""What a default run of the canonical walkers returns: the results of the
fastest schedule that is not pipelined, made by the fastest schedule that gives
those results bit for bit (the grouped and pipelined ones with equal teams).
"""
import numpy as np
import pytest

import pimc_gb300 as pgb
from pimc_gb300 import worldlines as wl

pytestmark = pytest.mark.gpu

MIXES = [(8, 96), (30, 37), (60, 30), (600, 20)]
PIPELINED = (5000, 5008, 5016, 6000, 6008, 6016)


def _run(num, nmax, schedule=0, steps=3):
    w = wl.workload_walkers(num=num, seed=0, nmin=8, nmax=nmax)
    W = pgb.Walkers(w["n"], w["m"], w["temperature"], w["side"], w["mbar"], w["tau"], w["lam"], seed=5,
                    threads_per_walker=schedule)
    W.init()
    W.run(steps)
    got = (W.stats_array().tobytes(), W.all_positions().tobytes())
    info = W.threads(), W.tuning()
    W.close()
    return got, info


def _group(schedule):
    """Schedules whose walkers have the same teams up to a CTA's size."""
    return [schedule] if schedule < 5000 else [t + schedule % 1000 for t in (5000, 6000, 7000, 8000)]


@pytest.mark.parametrize("num,nmax", MIXES)
def test_pipelined_times_do_not_choose_the_results(num, nmax):
    got, (picked, times) = _run(num, nmax)
    decide = {k: v for k, v in times.items() if k not in PIPELINED}
    results = min(decide, key=decide.get)
    assert picked in _group(results)
    # and the results are those of the schedule that decided
    assert got == _run(num, nmax, results)[0]


@pytest.mark.parametrize("num,nmax", MIXES)
@pytest.mark.parametrize("teams", [0, 8, 16])
def test_equal_teams_give_equal_results(num, nmax, teams):
    want = _run(num, nmax, 8000 + teams)[0]
    for schedule in (6000 + teams, 7000 + teams):
        assert _run(num, nmax, schedule)[0] == want
    if teams and num > 8:            # teams of at most eight warps: a smaller CTA holds them too
        assert _run(num, nmax, 5000 + teams)[0] == want
