"""The Gaussian-process kernels at the edges of their blocks, against the oracle."""
import numpy as np
import pytest

from pimc_gb300 import worldlines as wl


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [0.5, 1.5, 2.5])
@pytest.mark.parametrize("points,num_ptcl,num_slices", [(1, 1, 1), (33, 1, 31), (65, 3, 43), (700, 1, 257), (257, 5, 77)])
@pytest.mark.parametrize("side", [14.0, 2.5])
def test_chunks_points_and_images(pgb, oracle_lib, nu, points, num_ptcl, num_slices, side):
    """Remainders of points and chunks, and boxes that need images (side 2.5 in
    normalised coordinates) or not, beside coinciding points and one outside.
    FP64: within 1e-12 of the oracle, as elsewhere; mixed: FP32 kernel values,
    each within 2e-5 (an exponent up to 20 carries 20 2^-23, the separations and
    the polynomial as much again), of std sigma2 sum_k |w_k|."""
    from pimc_gb300 import PGB_MIXED
    from pimc_gb300.gp import GaussianProcess
    w = wl.workload_gp(points=points, num_ptcl=num_ptcl, num_slices=num_slices, seed=points, matern_nu=nu)
    w["params"]["side"] = [side] * 3
    w["params"]["periodic"] = [1, 0, 1]
    pos = w["pos"].copy()
    pos[0] = np.array(w["training"][0, :3]) * w["params"]["norm_scale"] + w["params"]["norm_offset"]
    pos[-1] = [40.0, -35.0, 21.0]
    p = w["params"]
    want = oracle_lib.gp_eval(w["training"], pos, **p)
    scale = p["standard_std"] * p["sigma2"] * np.abs(w["training"][:, 3]).sum()
    got = GaussianProcess(w["training"], **p)(pos)
    assert np.max(np.abs(got - want)) <= 1e-12 * max(scale, np.abs(want).max())
    mixed = GaussianProcess(w["training"], precision=PGB_MIXED, **p)
    for _ in range(2):                                    # the arrival counters return to 0
        assert np.max(np.abs(mixed(pos) - want)) <= 2e-5 * scale
