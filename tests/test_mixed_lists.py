"""Mixed S(q) and F(q,tau) on both sides of the rules that share the work out:
few and many vectors, short paths (many vectors a CTA) and long ones, odd
numbers of slices.  All forms against a NumPy correlation of the library's
FP64 densities.

Tolerance: an FP32 density is off by at most n 2^-21 (phase in turns to 2^-24,
FP32 sine, n terms added), a product of two, |rho| <= n, by 2 n^2 2^-21, and the
64-term FP32 sums by another 64 2^-24 n^2.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 4, 9, 62, 257])
@pytest.mark.parametrize("nq", [1, 150, 299, 300, 400])
def test_few_and_many(pgb, m, nq):
    n = 8
    L = pgb.worldlines.box_side(n)
    cfg = pgb.worldlines.seeded_worldlines(n, m, L, 6.0596, 0.004, m)
    a = pgb.Action(L, m, n, 0.004, 6.0596, precision=pgb.PGB_MIXED)
    a.load(cfg)
    rng = np.random.default_rng(nq)
    q = np.ascontiguousarray((2 * np.pi / L) * rng.integers(-4, 5, (nq, 3)))
    z = a.rhoq(q)
    z = z[..., 0] + 1j * z[..., 1]
    F = np.stack([(z * np.conj(np.roll(z, -k, 1))).real.sum(1) for k in range(m // 2 + 1)], 1) / (n * m)
    tol = n * (2.0 ** -20 + 2.0 ** -18)
    assert np.max(np.abs(a.isf(q) - F)) <= tol
    assert np.max(np.abs(a.ssf(q) - F[:, 0])) <= tol
