"""Mixed-form estimator kernels at the edges of their blocks: the slice sums
against those of another split, S(q) and F(q,tau) against the FP64 form with
the 2e-4 that the mixed form is held to at other sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(pgb, n, m, seed):
    """Particles on a jittered grid: the FP64 tables and the FP32 formula agree
    where pairs do not overlap."""
    L = pgb.worldlines.box_side(n)
    rng = np.random.default_rng(seed)
    g = int(np.ceil(n ** (1 / 3)))
    site = np.stack(np.unravel_index(rng.permutation(g ** 3)[:n], (g, g, g)), 1)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, seed)
    r = (site + 0.5 + rng.uniform(-0.1, 0.1, (n, 3))) * (L / g) - 0.5 * L
    cfg["pos"] = np.ascontiguousarray(r[None] + rng.normal(0, 0.15, (m, n, 3)))
    cfg["pos"] -= L * np.floor(cfg["pos"] / L + 0.5)
    return cfg, L


def _pair(pgb, cfg, L, m, n, action="gsf"):
    out = []
    for prec in (pgb.PGB_MIXED, pgb.PGB_FP64):
        a = pgb.Action(L, m, n, 0.004, 6.0596, action=action, precision=prec)
        a.load(cfg)
        out.append(a)
    return out


# Slice sums (vint g2 r1 r2 d1 d2 kin xch over all slices, GSF) of the kernel
# with one CTA of 128 threads a slice, whose Kahan and FP32 sums fix an order:
# another split of the beads over CTAs has to keep it.
SUMS = {
    2: [-49.735445022583008, 98788.708934783936, 1009.2682449892163, 1079293.2412614822, 91.598781434819102, 107062.18630129099, 1.9386417083442211, 1.4057473064167425],
    33: [-3060.8385303653777, 46764611.077749252, 33723.85898861289, 560415916.21838379, 6169.4458121024072, 46026592.587162614, 34.763348167587537, 17.556033166067209],
    64: [-11696.943558748811, 199991.27559041977, 2269.1863121539354, 933092.34151771665, 211.75342033756897, 161422.0026258342, 73.050967327319086, 36.964556362276198],
    65: [995.95173703785986, 239983272.92366529, -39783.144226133823, 693426965.09640503, 20163.7361680381, 192759949.67552829, 71.563012073864229, 34.47162638532609],
    129: [-17442.85357647785, 72184338.249285698, 12268.204911917448, -77302076.830518723, 14477.931989169214, 44164718.186417624, 141.35406089155003, 72.126115415230743],
}


@pytest.mark.parametrize("n", sorted(SUMS))
def test_slice_sums_keep_their_order(pgb, n):
    """The FP32 parts equal bit for bit; adding eight slices in FP64 is within 1e-14."""
    cfg, L = _path(pgb, n, 8, n)
    a, _ = _pair(pgb, cfg, L, 8, n)
    e = a.energy()
    for _ in range(2):                                    # the arrival counters return to 0
        t = a.slice_terms()
        got = np.array([t[k].sum() for k in ("vint", "g2", "r1", "r2", "d1", "d2", "kin", "xch")])
        scale = np.array([np.abs(t[k]).sum() for k in ("vint", "g2", "r1", "r2", "d1", "d2", "kin", "xch")])
        assert np.all(np.abs(got - SUMS[n]) <= 1e-14 * scale)
    # the energy asks for less (the potential of each pair once on even slices)
    # and finds the same potential: its second column is vint / M + tail
    tail = n * n / L ** 3 * a.table_info()[2]
    vint = a.slice_terms()["vint"][::2].sum() / 4 + tail
    assert abs(e[3] - vint) <= 1e-14 * (scale[0] + abs(tail))


@pytest.mark.parametrize("n,m,nq", [(3, 2, 1), (5, 30, 17), (40, 62, 130), (9, 64, 9), (20, 67, 33), (6, 250, 70),
                                    (2, 1030, 3), (2, 15400, 2)])
def test_correlation(pgb, n, m, nq):
    cfg, L = _path(pgb, n, m, n + m)
    q = (2 * np.pi / L) * np.random.default_rng(nq).integers(-6, 7, (nq, 3))
    a, o = _pair(pgb, cfg, L, m, n, "primitive")
    assert np.max(np.abs(a.isf(q) - o.isf(q))) <= 2e-4
    assert np.max(np.abs(a.ssf(q) - o.ssf(q))) <= 2e-4
