"""The calls that a user of pimc_gb300 makes, as measured cases.

Each case has a "kind":

  move       one Metropolis decision of the drop-in ActionBase: the bead
             actions of a diagonal move's range before and after the beads
             move, the beads put back, and the same beads as single trials
  trials     many independent single-bead trial displacements on device buffers
  sample     one estimator sample of a path whose positions come from the host
  scatter    S(q) and F(q,tau) of a path whose positions are on the device
  gp         the Gaussian-process external potential over a path's beads
  plain      steps of the host-driven FP64 worm algorithm
  worm       steps of the device worm walkers
  canonical  sweeps of the canonical walkers
  serving    jobs through the continuous-batching server, until all are done

Paths come from the package's seeded worldlines with exchange cycles; sizes
from its workloads, tests and bench.
"""
import math

import numpy as np
import torch

import pimc_gb300 as pgb
from pimc_gb300 import worldlines as wl
from pimc_gb300.gp import GaussianProcess

TAU = wl.TAU
LAM = wl.LAMBDA_HE4


def listed():
    return [
        # the plug-in's smallest call: a bisection range of a 64-particle path,
        # an open worm in it, FP64 (the default precision)
        dict(name="move_fp64", kind="move", n=64, m=124, k=31, action="gsf", precision="fp64"),
        # the pair-action workload: a million trial displacements, N = 256, GSF
        dict(name="trials_1e6", kind="trials", n=256, m=250, k=1000000, action="gsf", precision="mixed"),
        # every estimator of one sample, FP64 and primitive action, as the
        # plug-in's estimators ask for it on an ordinary path
        dict(name="sample_fp64", kind="sample", n=64, m=124, action="primitive", precision="fp64", qmax=2.0),
        # the same on the large GSF path in mixed precision
        dict(name="sample_mixed", kind="sample", n=256, m=250, action="gsf", precision="mixed", qmax=2.0),
        # the F(q,tau) workload: 2048 lattice q, tensor-core correlation
        dict(name="scatter_tc", kind="scatter", n=512, m=512, nq=2048, q="lattice", mode=1, precision="mixed"),
        # F(q,tau) at ragged sizes with shell q (not lattice vectors), CUDA cores
        dict(name="scatter_ragged", kind="scatter", n=101, m=190, nq=333, q="shells", mode=0, precision="mixed"),
        # FP64 F(q,tau), the form the plain runs are checked with
        dict(name="scatter_fp64", kind="scatter", n=128, m=250, nq=300, q="lattice", mode=0, precision="fp64"),
        # the Gaussian-process potential: 64 x 64 beads, 16384 training points
        dict(name="gp_mixed", kind="gp", points=16384, n=64, m=64, nu=2.5, precision="mixed"),
        # the host-driven form at its own workload: N = 16 at 2 K
        dict(name="plain_n16", kind="plain", n=16, t=2.0, steps=10),
        # the bosonic walkers: 1024 paths, N 8..128, T 1..4 K, and a checkpoint
        dict(name="worm_1024", kind="worm", num=1024, nmin=8, nmax=128, tmin=1.0, tmax=4.0, window=1,
             staging=False, sweeps=4, state=True),
        # the canonical walkers on the same mix (autotuned schedule)
        dict(name="canonical_1024", kind="canonical", num=1024, nmin=8, nmax=128, tmin=1.0, tmax=4.0,
             sweeps=10, state=False),
        # grand-canonical jobs of mixed sizes served together
        dict(name="serving_32", kind="serving", jobs=32, nmin=8, nmax=96, tmin=1.0, tmax=4.0, sweeps=12),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["move", "trials", "sample", "scatter", "gp", "plain", "worm", "canonical", "serving"])
    precision = rng.choice(["fp64", "mixed"])
    action = rng.choice(["primitive", "gsf", "li_broughton"])
    if kind == "move":
        return dict(kind=kind, n=_logint(rng, 9, 256), m=2 * _logint(rng, 20, 125),
                    k=rng.choice([1, 3, 7, 15, 31]), action=action, precision=precision)
    if kind == "trials":
        # FP64 trials are the check, mixed ones the production form
        most = 20000 if precision == "fp64" else 1000000
        return dict(kind=kind, n=_logint(rng, 16, 128 if precision == "fp64" else 256), m=2 * _logint(rng, 16, 125),
                    k=_logint(rng, 100, most), action=action, precision=precision)
    if kind == "sample":
        return dict(kind=kind, n=_logint(rng, 8, 128 if precision == "fp64" else 256), m=2 * _logint(rng, 8, 125),
                    action=action, precision=precision, qmax=rng.choice([1.0, 1.5, 2.0]))
    if kind == "scatter":
        if precision == "mixed" and rng.random() < 0.5:
            return dict(kind=kind, n=_logint(rng, 16, 512), m=rng.choice([128, 256, 384, 512]),
                        nq=_logint(rng, 16, 2048), q="lattice", mode=1, precision=precision)
        return dict(kind=kind, n=_logint(rng, 16, 512 if precision == "mixed" else 160), m=2 * _logint(rng, 8, 125),
                    nq=_logint(rng, 16, 1024 if precision == "mixed" else 400), q=rng.choice(["lattice", "shells"]),
                    mode=0, precision=precision)
    if kind == "gp":
        return dict(kind=kind, points=_logint(rng, 128, 16384 if precision == "mixed" else 2048),
                    n=_logint(rng, 4, 64), m=2 * _logint(rng, 4, 32), nu=rng.choice([0.5, 1.5, 2.5]),
                    precision=precision)
    if kind == "plain":
        return dict(kind=kind, n=rng.randint(8, 24), t=rng.uniform(1.5, 4.0), steps=rng.randint(4, 10))
    if kind == "serving":
        return dict(kind=kind, jobs=_logint(rng, 4, 32), nmin=8, nmax=_logint(rng, 16, 96), tmin=1.0, tmax=4.0,
                    sweeps=rng.randint(4, 12))
    num, nmax = _logint(rng, 8, 600), _logint(rng, 16, 128)
    if kind == "worm":
        return dict(kind=kind, num=num, nmin=8, nmax=nmax, tmin=1.0, tmax=4.0, window=rng.choice([-1, 1]),
                    staging=rng.random() < 0.3, sweeps=rng.randint(1, 4), state=True)
    return dict(kind=kind, num=num, nmin=8, nmax=nmax, tmin=1.0, tmax=4.0, sweeps=rng.randint(1, 10),
                state=num * nmax < 8000)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(seed, salt):
    return np.random.Generator(np.random.Philox(key=[seed, salt]))


def _prec(case):
    return pgb.PGB_MIXED if case["precision"] == "mixed" else pgb.PGB_FP64


def _wrap(r, side):
    return r - side * np.floor(r / side + 0.5)


def _path(n, m, seed):
    """A closed path with exchange cycles: particles on a jittered grid (a
    liquid has no overlaps), beads jittered about them, and two cycles."""
    L = wl.box_side(n)
    rng = _rng(seed, 1)
    g = math.ceil(n ** (1.0 / 3.0))
    site = np.stack(np.unravel_index(rng.permutation(g ** 3)[:n], (g, g, g)), 1)
    centre = (site + 0.5 + rng.uniform(-0.15, 0.15, (n, 3))) * (L / g) - 0.5 * L
    cfg = wl.seeded_worldlines(n, m, L, LAM, TAU, seed)
    jit = rng.normal(0.0, math.sqrt(2.0 * LAM * TAU), size=(m, n, 3))
    cfg["pos"] = np.ascontiguousarray(_wrap(centre[None] + jit, L))
    perm = np.arange(n)
    for cyc in ((1, 4), (2, 5, 7)):
        if max(cyc) < n:
            perm[list(cyc)] = np.roll(cyc, -1)
            cfg = wl.permute(cfg, [cyc])
    return cfg, L, perm


def _open(cfg, m):
    """The worm's head and tail on the last particle, a sixth of the path apart."""
    p = cfg["pos"].shape[1] - 1
    return wl.open_worm(cfg, (m // 3, p), (m // 2, p))


def _moves(case, cfg, L, seed):
    """The beads of a diagonal move on particle 3 and where it puts them."""
    m, k = case["m"], min(case["k"], case["m"] - 3)
    s0 = m // 3 - k // 2
    beads = np.stack([np.arange(s0, s0 + k) % m, np.full(k, 3)], 1).astype(np.int32)
    old = np.ascontiguousarray(cfg["pos"][beads[:, 0], beads[:, 1]])
    new = _wrap(old + _rng(seed, 2).normal(0.0, math.sqrt(LAM * TAU), (k, 3)), L)
    return beads, old, np.ascontiguousarray(new)


def _trials(case, cfg, L, seed):
    n, m, k = case["n"], case["m"], case["k"]
    rng = _rng(seed, 3)
    beads = np.stack([rng.integers(0, m, k), rng.integers(0, n, k)], 1).astype(np.int32)
    step = 0.04 * 2.0 * math.sqrt(math.pi * LAM * m * TAU)
    pos = _wrap(cfg["pos"][beads[:, 0], beads[:, 1]] + rng.uniform(-step, step, (k, 3)), L)
    return beads, np.ascontiguousarray(pos)


def _qvectors(case, L, seed):
    if case["kind"] == "sample":
        return pgb.qvectors("max_float", "%g 0 0" % case["qmax"], [L, L, L])
    if case["q"] == "lattice":
        q = wl.isf_qvectors(L, count=case["nq"], seed=seed, qmax=4.0)[0]
        while len(q) < case["nq"]:                       # small boxes have fewer lattice vectors
            q = np.concatenate([q, q])[:case["nq"]]
        return np.ascontiguousarray(q)
    q = pgb.qvectors_shells(0.2, 4.0, sphere=True)[0]
    return np.ascontiguousarray(q[_rng(seed, 4).permutation(len(q))[:case["nq"]]])


def _gp(case, seed):
    w = wl.workload_gp(points=case["points"], num_ptcl=case["n"], num_slices=case["m"], seed=seed,
                       matern_nu=case["nu"])
    return w["training"], w["params"], w["pos"]


def _mix(case):
    # one mix of sizes for a case, whatever the seed of its chains
    return wl.workload_walkers(num=case["num"], seed=0, nmin=case["nmin"], nmax=case["nmax"], tmin=case["tmin"],
                               tmax=case["tmax"])


def _jobs(case, seed):
    rng = _rng(7, 5)                                     # one mix of jobs; their chains come from the seed
    return [dict(n=int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]))))),
                 temperature=float(rng.uniform(case["tmin"], case["tmax"])), mu=float(rng.uniform(-10.0, 0.0)),
                 sweeps=case["sweeps"], seed=1000 * seed + i) for i in range(case["jobs"])]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("move", "trials", "sample", "scatter"):
        n, m = case["n"], case["m"]
        cfg, L, _ = _path(n, m, seed)
        if kind == "move":
            cfg = _open(cfg, m)
        a = pgb.Action(L, m, n, TAU, LAM, action=case.get("action", "primitive"), precision=_prec(case))
        a.load(cfg)
        s["a"] = a
        if kind == "move":
            s["beads"], s["old"], s["new"] = _moves(case, cfg, L, seed)
        elif kind == "trials":
            beads, pos = _trials(case, cfg, L, seed)
            s["beads"], s["pos"] = torch.from_numpy(beads).cuda(), torch.from_numpy(pos).cuda()
            s["out"] = torch.empty(case["k"], dtype=torch.float64, device="cuda")
            s["work"] = torch.empty(2 * case["k"], dtype=torch.float64, device="cuda")
        elif kind == "sample":
            s["pos"], s["q"] = cfg["pos"], _qvectors(case, L, seed)
        else:
            # positions in the device layout of pgb_load_positions_device_async: [M][3][Ne]
            s["pos"] = torch.from_numpy(np.ascontiguousarray(cfg["pos"].transpose(0, 2, 1))).cuda()
            s["q"] = torch.from_numpy(_qvectors(case, L, seed)).cuda()
            s["isf"] = torch.empty((case["nq"], m // 2 + 1), dtype=torch.float64, device="cuda")
            s["ssf"] = torch.empty(case["nq"], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    elif kind == "gp":
        train, params, s["pos"] = _gp(case, seed)
        s["gp"] = GaussianProcess(train, precision=_prec(case), **params)
    elif kind == "plain":
        n, m = case["n"], wl.even_slices(case["t"], TAU)
        L = wl.box_side(n)
        a = pgb.Action(L, m, 2 * n, 1.0 / (m * case["t"]), LAM)
        a.load(wl.seeded_worldlines(n, m, L, LAM, TAU, seed, extent=2 * n))
        a.plain_seed(seed % (1 << 31) + 1)
        s["a"] = a
        s["args"] = dict(mbar=wl.default_mbar(n, L ** 3, LAM, TAU, m), temperature=case["t"],
                         initial_num_particles=n, window=1, mu=0.0)
    elif kind == "worm":
        w = _mix(case)
        W = pgb.WormWalkers(w["n"], w["m"], w["side"], w["mbar"], w["tau"], w["lam"], window=case["window"],
                            mu=-2.0, seed=seed, diagonal_move=int(case["staging"]))
        W.seed_device(seed)
        W.equilibrate(20)
        s["walkers"] = W
        if case["state"]:
            s["image"] = torch.empty(W.state_bytes(), dtype=torch.uint8, pin_memory=True).numpy()
    elif kind == "canonical":
        w = _mix(case)
        W = pgb.Walkers(w["n"], w["m"], w["temperature"], w["side"], w["mbar"], w["tau"], w["lam"], seed=seed)
        W.init()
        W.run(3)
        s["walkers"] = W
    else:
        s["server"] = pgb.Server(2e9, max_active=64, sweeps_per_round=4, bin_sweeps=4, grand_canonical=True)
        s["jobs"] = _jobs(case, seed)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _run_worm(s):
    W = s["walkers"]
    W.run(s["case"]["sweeps"])
    st = W.stats()
    out = {k: st[k].copy() for k in W.STATS_DTYPE.names if k != "pad"}
    if s["case"]["state"]:
        W.get_state(s["image"])
        # positions, links and bead counts, in the image's order
        nb = int((W.m.astype(np.int64) * W.capacity).sum())
        ns = int(W.m.sum())
        at = np.cumsum([0, 16 * nb, 4 * nb, 4 * nb, 4 * ns])
        part = [s["image"][at[i]:at[i + 1]] for i in range(4)]
        out.update(pos=part[0].view(np.float32), next=part[1].view(np.int32), prev=part[2].view(np.int32),
                   counts=part[3].view(np.int32))
    return out


def _run_serving(s):
    srv, ids, bins = s["server"], [], []
    for j in s["jobs"]:
        ids.append(srv.submit(**j))
    while True:
        active, queued = srv.step()
        bins += srv.bins()
        if not active and not queued:
            break
    bins.sort(key=lambda b: (b["job"], b["bin"]))
    return dict(job=np.array([b["job"] - ids[0] for b in bins]), bin=np.array([b["bin"] for b in bins]),
                energy=np.array([b["energy"] for b in bins]), samples=np.array([b["samples"] for b in bins]),
                sweeps=np.array([srv.job(i)["sweeps_done"] for i in ids]))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "move":
        a = s["a"]
        before, u0 = a.bead_actions(s["beads"])
        a.update_beads(s["beads"], s["new"])
        after, u1 = a.bead_actions(s["beads"])
        a.update_beads(s["beads"], s["old"])
        return dict(before=before, after=after, change=u1 - u0, single=a.trial_actions(s["beads"], s["new"]))
    if kind == "trials":
        a = s["a"]
        a._chk(a.lib.pgb_trial_actions_device_async(a.h, s["beads"].data_ptr(), s["pos"].data_ptr(), case["k"], 1,
                                                    pgb.PGB_ACTION_FULL, s["out"].data_ptr(), s["work"].data_ptr()))
        return s["out"]
    if kind == "sample":
        a = s["a"]
        a.update_positions(s["pos"])
        return dict(energy=a.energy(), virial=a.virial(), ssf=a.ssf(s["q"]), isf=a.isf(s["q"]),
                    pair_correlation=a.pair_correlation(), superfluid=a.superfluid(),
                    cycles=a.permutation_cycles())
    if kind == "scatter":
        a = s["a"]
        a._chk(a.lib.pgb_load_positions_device_async(a.h, s["pos"].data_ptr()))
        a._chk(a.lib.pgb_ssf_device_async(a.h, s["q"].data_ptr(), case["nq"], s["ssf"].data_ptr()))
        a._chk(a.lib.pgb_isf_device_async(a.h, s["q"].data_ptr(), case["nq"], case["mode"], s["isf"].data_ptr()))
        return dict(ssf=s["ssf"], isf=s["isf"])
    if kind == "gp":
        return s["gp"](s["pos"])
    if kind == "plain":
        a = s["a"]
        r = a.plain_worm_run(case["steps"], **s["args"])
        p = a.path()
        return dict(energies=r["energies"], num_particles=r["num_particles"], attempted=np.array(r["attempted"]),
                    accepted=np.array(r["accepted"]), bead_updates=r["bead_updates"], diagonal=r["diagonal"],
                    pos=p["pos"], next=p["next"], prev=p["prev"], on=p["on"], worm=p["worm"])
    if kind == "worm":
        return _run_worm(s)
    if kind == "canonical":
        W = s["walkers"]
        W.run(case["sweeps"])
        st = W.stats_array()
        out = {k: st[k].copy() for k in W.STATS_DTYPE.names}
        out["sweeps"] = W.sweeps_done().astype(np.int64)
        if case["state"]:
            out["pos"] = W.all_positions()
        return out
    return _run_serving(s)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
PAIR_V, PAIR_VG = 40.0, 52.0          # a pair's potential; with its gradient


def work(case):
    kind = case["kind"]
    n, m = case.get("n", 0), case.get("m", 0)
    corr = {"primitive": 0.0, "gsf": 0.5, "li_broughton": 1.0}[case.get("action", "primitive")]
    if kind == "move":
        # the moved beads' pairs before and after, and the slice's pair forces
        # for the gradient term; the partners' positions read once
        k = min(case["k"], m - 3)
        return dict(bytes=24.0 * k * n + 24.0 * k * 5, flops=k * (2.0 * PAIR_VG * (n - 1) + corr * PAIR_VG * n * n / 2))
    if kind == "trials":
        k = case["k"]
        beads = min(k, m * n)         # a bead's current action serves all its trials
        return dict(bytes=40.0 * k + 24.0 * m * n,
                    flops=(k + beads) * (n - 1.0) * (PAIR_V + corr * (PAIR_VG - PAIR_V)) + corr * PAIR_VG * m * n * n / 2)
    if kind == "sample":
        nq = 4.0 / 3.0 * math.pi * (case["qmax"] * wl.box_side(n) / (2.0 * math.pi)) ** 3
        return dict(bytes=24.0 * m * n + 16.0 * m * n + 8.0 * nq * (m / 2 + 2),
                    flops=m * n * (n - 1) / 2.0 * (PAIR_VG + 30.0) + nq * m * (n * 14.0 + 20.0 * math.log2(m)))
    if kind == "scatter":
        nq = case["nq"]
        corr_flops = 20.0 * math.log2(m) if case["mode"] == 0 else 4.0 * m
        return dict(bytes=24.0 * m * n + 24.0 * nq + 8.0 * nq * (m / 2 + 2), flops=nq * m * (n * 14.0 + corr_flops))
    if kind == "gp":
        pts = n * m
        return dict(bytes=32.0 * pts + 32.0 * case["points"], flops=40.0 * pts * case["points"])
    if kind == "plain":
        # one update a Metropolis decision over about half an update length
        mm = wl.even_slices(case["t"], TAU)
        moved = max(100, n * mm / 32.0) * 16.0
        return dict(bytes=2.0 * 40.0 * n * mm, flops=case["steps"] * (moved * 2 * (n - 1) + mm * n * n / 2.0) * PAIR_V)
    if kind == "serving":
        jobs = _jobs(case, 0)
        nn = np.array([j["n"] for j in jobs], float)
        mm = np.array([max(4, 2 * round(0.5 / (j["temperature"] * TAU))) for j in jobs], float)
        cap, moved, sweeps = 2 * nn + 8, 0.25, case["sweeps"]
    else:
        w = _mix(case)
        nn, mm = w["n"].astype(float), w["m"].astype(float)
        cap, moved, sweeps = (2 * nn + 8, 0.25, case["sweeps"]) if kind == "worm" else (nn, 0.5, case["sweeps"])
    per_bead = 24.0 if kind != "canonical" else 16.0
    pairs = moved * mm * nn * 2 * (nn - 1) + mm * nn * (nn - 1) / 2
    return dict(bytes=float(2 * per_bead * (mm * cap).sum()), flops=float(sweeps * PAIR_V * pairs.sum()))


# ---------------------------------------------------------------------------
# the same in 64 bits, from the formulas (the random chains have none)
# ---------------------------------------------------------------------------
AZIZ = dict(rm=2.9673, A=0.5448504E6, eps=10.8, alpha=13.353384, D=1.241314, C6=1.3732412, C8=0.4253785, C10=0.1781)


class _Aziz:
    """V, V'/r and V'' of the 1979 Aziz potential: at r for the mixed form, at
    the grid point at or below r for the FP64 form, whose tables are on a grid
    of step 1e-6 rm with zero at its first point and beyond its end."""

    def __init__(self, L, table):
        self.table = table
        if table:
            self.dr = 1.0e-6 * AZIZ["rm"]
            n = int(math.sqrt(0.75 * L * L) / self.dr)
            grid = np.concatenate([[0.0], np.cumsum(np.full(n - 1, self.dr))])
            self.grid = torch.from_numpy(grid).cuda()

    def __call__(self, r2, second=False):
        p = AZIZ
        r = torch.sqrt(r2)
        at, live = r, r > 0
        if self.table:
            k = (r / self.dr).long()
            live = (k > 0) & (k < len(self.grid))
            at = self.grid[k.clamp(1, len(self.grid) - 1)]
        ix = p["rm"] / torch.where(live, at, torch.full_like(at, p["rm"]))
        e = p["A"] * torch.exp(-p["alpha"] / ix)
        t = (p["D"] * ix - 1.0).clamp(min=0.0)
        F = torch.exp(-t * t)
        dF = 2.0 * p["D"] * ix ** 2 * t * F
        p0 = p["C6"] * ix ** 6 + p["C8"] * ix ** 8 + p["C10"] * ix ** 10
        p1 = 6 * p["C6"] * ix ** 7 + 8 * p["C8"] * ix ** 9 + 10 * p["C10"] * ix ** 11
        zero = torch.zeros_like(r)
        V = torch.where(live, p["eps"] * (e - p0 * F), zero)
        g = torch.where(live, p["eps"] / p["rm"] * (-p["alpha"] * e + p1 * F - p0 * dF) / r.clamp(min=1e-9), zero)
        if not second:
            return V, g
        p2 = 42 * p["C6"] * ix ** 8 + 72 * p["C8"] * ix ** 10 + 110 * p["C10"] * ix ** 12
        y = p["D"] * ix
        d2F = torch.where(t > 0, 2 * p["D"] * ix ** 3 * (2 * y ** 3 - 4 * y ** 2 - y + 2) * F, zero)
        d2 = p["eps"] / p["rm"] ** 2 * (p["alpha"] ** 2 * e - p2 * F + 2 * p1 * dF - p0 * d2F)
        return V, g, torch.where(live, d2, zero)


def _img(d, L):
    return d - L * torch.floor(d / L + 0.5)


def _factors(case):
    return {"primitive": ((1.0, 1.0), (0.0, 0.0), 1), "gsf": ((2 / 3, 4 / 3), (0.0, 2 / 9), 2),
            "li_broughton": ((1.0, 1.0), (1 / 12, 1 / 12), 2)}[case["action"]]


def _bead_action(case, pot, L, pos, on, cut, beads, at):
    """Potential action of beads[i] at at[i] with every other bead where it is.
    `cut`: the worm's (head, tail), whose pairs count half or, between them, not."""
    vf, gf, _ = _factors(case)
    out = []
    n = pos.shape[1]
    idx = torch.arange(n, device=pos.device)
    for i in range(0, len(beads), max(1, 4000000 // n)):
        b, x = beads[i:i + max(1, 4000000 // n)], at[i:i + max(1, 4000000 // n)]
        sl, p = b[:, 0], b[:, 1]
        P = pos[sl]
        other = on[sl] & (idx[None] != p[:, None])
        d = _img(P - x[:, None], L)
        V, g = pot((d * d).sum(-1))
        f = torch.ones_like(V)
        for s_, p_ in cut:
            f[(sl == s_)[:, None] & (idx == p_)[None]] *= 0.5
        U = torch.tensor(vf, device=pos.device, dtype=torch.float64)[sl % 2] * TAU * (V * f * other).sum(1)
        c = torch.tensor(gf, device=pos.device, dtype=torch.float64)[sl % 2]
        if max(gf) > 0:
            F2 = torch.where(other[..., None], g[..., None] * d, torch.zeros_like(d))
            o = _img(P - pos[sl, p][:, None], L)
            go = pot((o * o).sum(-1))[1]
            F3 = torch.where(other[..., None], _force(case, pot, L, pos, on)[sl] - go[..., None] * o, torch.zeros_like(d))
            T = (F2 * F2).sum((1, 2)) + 2.0 * (F2 * F3).sum((1, 2)) + (F2.sum(1) ** 2).sum(1)
            U = U + c * TAU ** 3 * LAM * T
        out.append(U)
    return torch.cat(out)


_held = {}


def _force(case, pot, L, pos, on):
    """Every active bead's force from its slice, kept while one path is asked about."""
    if _held.get("pos") is not pos:
        f = torch.zeros_like(pos)
        for t in range(pos.shape[0]):
            d = _img(pos[t][:, None] - pos[t][None], L)
            r2 = (d * d).sum(-1) + 1e3 * torch.eye(pos.shape[1], device=pos.device, dtype=torch.float64)
            g = pot(r2)[1] * on[t][None] * (1.0 - torch.eye(pos.shape[1], device=pos.device, dtype=torch.float64))
            f[t] = (g[..., None] * d).sum(1)
        _held.clear()
        _held.update(pos=pos, force=f)
    return _held["force"]


def _exact_actions(case, seed):
    cfg, L, _ = _path(case["n"], case["m"], seed)
    if case["kind"] == "move":
        cfg = _open(cfg, case["m"])
    pot = _Aziz(L, case["precision"] == "fp64")
    pos, on = torch.from_numpy(cfg["pos"]).cuda(), torch.from_numpy(cfg["on"]).cuda() > 0
    cut = [tuple(int(v) for v in cfg["worm"][:2]), tuple(int(v) for v in cfg["worm"][2:4])] if case["kind"] == "move" else []
    if case["kind"] == "trials":
        beads, new = _trials(case, cfg, L, seed)
        old = cfg["pos"][beads[:, 0], beads[:, 1]]
    else:
        beads, old, new = _moves(case, cfg, L, seed)
    b = torch.from_numpy(beads).cuda().long()
    u0, u1 = (_bead_action(case, pot, L, pos, on, cut, b, torch.from_numpy(x).cuda()) for x in (old, new))
    _held.clear()
    if case["kind"] == "trials":
        return u1 - u0
    return dict(before=u0, after=u1, change=float(u1.sum() - u0.sum()), single=u1 - u0)


def _densities(pos, q):
    """rho_q(t) [nq][M]."""
    out = []
    step = max(1, 30000000 // (pos.shape[0] * pos.shape[1]))
    for i in range(0, len(q), step):
        ph = torch.einsum("mnd,qd->qmn", pos, q[i:i + step])
        out.append(torch.complex(torch.cos(ph).sum(-1), torch.sin(ph).sum(-1)))
    return torch.cat(out)


def _structure(pos, q):
    m, n = pos.shape[:2]
    X = torch.fft.fft(_densities(pos, q), dim=1)
    F = torch.fft.ifft((X.real ** 2 + X.imag ** 2).to(torch.complex128), dim=1).real[:, :m // 2 + 1] / (n * m)
    return F[:, 0].contiguous(), F.contiguous()


def _exact_sample(case, seed):
    n, m = case["n"], case["m"]
    cfg, L, perm = _path(n, m, seed)
    vf, gf, period = _factors(case)
    pot = _Aziz(L, case["precision"] == "fp64")
    pos = torch.from_numpy(cfg["pos"]).cuda()
    perm = torch.from_numpy(perm).cuda()
    back = torch.argsort(perm)
    eye = torch.eye(n, device="cuda", dtype=torch.float64)

    def shift(x, up):                                    # the beads one link on (or back)
        y = torch.roll(x, -1 if up else 1, 0)
        y[-1 if up else 0] = x[0][perm] if up else x[-1][back]
        return y

    W = 5
    nxt, prv = [pos], [pos]
    for _ in range(W):
        nxt.append(shift(nxt[-1], True))
        prv.append(shift(prv[-1], False))
    up = [_img(nxt[g] - nxt[g - 1], L) for g in range(1, W + 1)]
    dn = [_img(prv[g] - prv[g - 1], L) for g in range(1, W + 1)]
    com, a, b = torch.zeros_like(pos), torch.zeros_like(pos), torch.zeros_like(pos)
    for g in range(W):
        if g:
            a, b = a + up[g - 1], b + dn[g - 1]
        com = com + (pos + a) + (pos + b)
    dev = _img(pos - com / (2.0 * W), L)
    kin = (up[0] ** 2).sum((1, 2))
    xch = (sum(up) * up[0]).sum((1, 2))
    vint, g2, r1, r2, d1, d2 = (torch.zeros(m, device="cuda", dtype=torch.float64) for _ in range(6))
    dsep = 0.5 * math.sqrt(3.0) * L / 50
    hist = torch.zeros(50, device="cuda", dtype=torch.float64)
    upper = torch.triu(torch.ones(n, n, device="cuda"), 1) > 0
    for t in range(m):
        d = _img(pos[t][:, None] - pos[t][None], L)
        rr = (d * d).sum(-1) + 1e3 * eye
        V, g, c2 = pot(rr, second=True)
        V, g, c2 = V * (1 - eye), g * (1 - eye), c2 * (1 - eye)
        F = (g[..., None] * d).sum(1)
        absg = g.abs()
        T = torch.einsum("ij,ija,ijb->iab", (c2 - absg) / rr, d, d) + absg.sum(1)[:, None, None] * torch.eye(3, device="cuda", dtype=torch.float64)
        TF = torch.einsum("iab,ib->ia", T, F)
        vint[t], g2[t] = V.sum() / 2, (F * F).sum()
        r1[t], r2[t] = (F * pos[t]).sum(), (TF * pos[t]).sum()
        d1[t], d2[t] = (F * dev[t]).sum(), (TF * dev[t]).sum()
        k = (torch.sqrt(rr[upper]) / dsep).long()
        hist += torch.bincount(k[k < 50], minlength=50).double()
    p = AZIZ
    y = p["rm"] / L
    vol = L ** 3
    tail = n * n / vol * 2 * math.pi * p["eps"] * -p["rm"] ** 3 * (p["C6"] * y ** 3 / 3 + p["C8"] * y ** 5 / 5 + p["C10"] * y ** 7 / 7)
    odd = torch.arange(m, device="cuda") % 2
    VF, GF = (torch.tensor(f, device="cuda", dtype=torch.float64)[odd] for f in (vf, gf))
    S = lambda x: float(x.sum())  # noqa: E731
    kn = 0.25 / (LAM * TAU) / (TAU * m)
    t1, t2 = S(GF * TAU ** 3 * g2) * LAM / (TAU * m), S(VF * vint + 3 * GF * TAU ** 2 * LAM * g2) / m
    K = -S(kin) * kn + 1.5 / TAU * n + t1
    Vt = t2 - t1 + tail
    energy = [K, Vt, 0.0, S(vint[::period]) / (m // period) + tail, K + Vt, K + Vt, K / n, Vt / n, (K + Vt) / n]
    beta = m * TAU
    T1, T2 = 1.5 * n / (W * TAU), -S(xch) / (4.0 * W * TAU ** 2 * LAM * m)
    T3, T4 = S(VF * TAU * d1) / (2 * beta), S(2 * GF * TAU ** 3 * LAM * d2) / beta
    vop = S(vint[::2]) / (0.5 * m) + tail
    press = (3 * n - S(kin) / (2 * LAM * TAU * m) - S(VF * TAU * r1 + 2 * GF * TAU ** 3 * LAM * r2) / (2.0 * m)) / (3 * TAU * vol)
    therm = -S(kin) * kn + 1.5 / TAU * n + t2 + tail
    ecv = T1 + T2 + T3 + T4 + t2 + tail
    kcv = T1 + T2 + T3 + T4 + S(GF * TAU ** 3 * LAM * g2) / (0.5 * beta)
    dE = ((-T1 - 2 * T2 + 2 * T4) / TAU + S(6 * GF * TAU * LAM * g2) / m) * beta * beta / m
    virial = [ecv - vop + ecv * beta * dE, kcv, vop, ecv - kcv, ecv, ecv, (ecv - vop) / n, kcv / n, vop / n, (ecv - kcv) / n,
              ecv / n, ecv * therm * beta ** 2, ecv * beta, dE, ecv * therm * beta ** 2 * ecv * beta, 0.0,
              ecv * therm * beta ** 2 * dE, therm, press]
    e = torch.arange(51, device="cuda", dtype=torch.float64) * dsep
    gr = (n - 1.0) / n * hist / max(S(hist), 1.0) * 0.5 * (3 / (2 * math.pi) * vol) / (e[1:] ** 3 - e[:-1] ** 3)
    w = up[0].sum((0, 1))
    sf = torch.zeros(26, device="cuda", dtype=torch.float64)
    sf[0], sf[1:4] = (w * w).sum() / n, (w / L) ** 2
    sf[4:25] = ((w[2] / L - torch.arange(-10, 11, device="cuda")).abs() < 0.2).double()
    area = (pos[..., 0] * nxt[1][..., 1] - nxt[1][..., 0] * pos[..., 1]).sum()
    sf[25] = area ** 2 / (pos[..., :2] * nxt[1][..., :2]).sum()
    cyc = np.zeros(40)
    seen, pm = set(), perm.cpu().numpy()
    for i in range(n):
        j, length = i, 0
        while j not in seen:
            seen.add(j)
            j, length = int(pm[j]), length + 1
        if 0 < length <= 40:
            cyc[length - 1] += length / n
    ssf, isf = _structure(pos, torch.from_numpy(_qvectors(case, L, seed)).cuda())
    return dict(energy=np.array(energy), virial=np.array(virial), ssf=ssf, isf=isf, pair_correlation=gr, superfluid=sf,
                cycles=cyc)


def _exact_gp(case, seed):
    train, p, pos = _gp(case, seed)
    tr = torch.from_numpy(train).cuda()
    r = (torch.from_numpy(pos).cuda() - torch.tensor(p["norm_offset"], device="cuda", dtype=torch.float64)) / torch.tensor(
        p["norm_scale"], device="cuda", dtype=torch.float64)
    out = []
    for i in range(0, len(r), 256):
        s = tr[None, :, :3] - r[i:i + 256, None]
        s = _img(s, p["side"][0]) / torch.tensor(p["ell"], device="cuda", dtype=torch.float64)
        x = math.sqrt(2 * case["nu"]) * torch.sqrt((s * s).sum(-1))
        poly = {0.5: 1.0, 1.5: 1 + x, 2.5: 1 + x + x * x / 3}[case["nu"]]
        out.append((poly * torch.exp(-x) * tr[:, 3]).sum(1))
    return p["standard_mean"] + p["standard_std"] * (p["mean"] + p["sigma2"] * torch.cat(out))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("move", "trials"):
        return _exact_actions(case, seed)
    if kind == "sample":
        return _exact_sample(case, seed)
    if kind == "scatter":
        cfg, L, _ = _path(case["n"], case["m"], seed)
        ssf, isf = _structure(torch.from_numpy(cfg["pos"]).cuda(), torch.from_numpy(_qvectors(case, L, seed)).cuda())
        return dict(ssf=ssf, isf=isf)
    return _exact_gp(case, seed) if kind == "gp" else None
