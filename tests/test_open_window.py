"""The centroid window's terms on a path with an open worldline: a walk that
meets an open end stays there for the rest of the window, in both precisions.
Against a NumPy walk, with the forces of the FP64 tables.

Tolerance: FP64 1e-12 of the sums of magnitudes (some hundred terms of a few
roundings each); mixed 2e-4 of them, as the FP32 forces are held to elsewhere.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = 5


def _walk(cfg, link, s, p, L):
    """Displacements to the 0th .. W-th neighbour along link."""
    at, d, out = (s, p), np.zeros(3), [np.zeros(3)]
    for _ in range(W):
        nx = tuple(cfg[link][at]) if at[0] >= 0 else at
        if nx[0] >= 0:
            step = cfg["pos"][nx] - cfg["pos"][at]
            d = d + step - L * np.floor(step / L + 0.5)
        at = nx
        out.append(d)
    return out


@pytest.mark.parametrize("head,tail", [((4, 3), (6, 3)), ((4, 3), (11, 3)), ((13, 3), (4, 3))])
@pytest.mark.parametrize("action", ["primitive", "gsf"])
def test_window(pgb, head, tail, action):
    n, m, L = 4, 16, 7.0
    rng = np.random.default_rng(2)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, 1)
    site = np.array([[-1.7, -1.7, -1.7], [1.7, 1.7, -1.7], [1.7, -1.7, 1.7], [-1.7, 1.7, 1.7]])
    cfg["pos"] = np.ascontiguousarray(site[None] + rng.normal(0, 0.25, (m, n, 3)))
    cfg = pgb.worldlines.open_worm(cfg, head, tail)
    acts = [pgb.Action(L, m, n, 0.004, 6.0596, action=action, precision=q, virial_window=W) for q in (pgb.PGB_FP64, pgb.PGB_MIXED)]
    for a in acts:
        a.load(cfg)
    want, scale = np.zeros((2, m)), np.zeros((2, m))
    for s in range(m):
        live = [i for i in range(n) if cfg["on"][s, i]]
        for i in live:
            d = np.array([cfg["pos"][s, i] - cfg["pos"][s, j] for j in live if j != i])
            d -= L * np.floor(d / L + 0.5)
            F = acts[0].gradV_batch(d).sum(0) if len(d) else np.zeros(3)
            fwd, back = _walk(cfg, "next", s, i, L), _walk(cfg, "prev", s, i, L)
            delta = -(sum(fwd[:W]) + sum(back[:W])) / (2 * W)
            delta -= L * np.floor(delta / L + 0.5)
            terms = F @ delta, fwd[W] @ fwd[1]
            want[:, s] += terms
            scale[:, s] += np.abs(F) @ np.abs(delta), np.abs(fwd[W]) @ np.abs(fwd[1])
    scale = np.maximum(scale, scale.max(1, keepdims=True))
    for a, tol in zip(acts, (1e-12, 2e-4)):
        t = a.slice_terms()
        got = np.stack([t["d1"], t["xch"]])
        assert np.all(np.abs(got - want) <= tol * scale)
