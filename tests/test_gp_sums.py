"""The mixed Gaussian-process form adds its chunks' parts in FP64: parts that
FP64 holds together and a pair of floats does not.  Every training point lies
on the inference point, so that each kernel value is 1 and the sum is that of
the weights, one a chunk of 32."""
import numpy as np
import pytest

from pimc_gb300 import PGB_MIXED
from pimc_gb300.gp import GaussianProcess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 130, 300])
def test_parts_in_fp64(count):
    chunks = 70
    train = np.zeros((32 * chunks, 4))
    train[::32, 3] = 2.0 ** -50
    train[0, 3] = 1.0
    train[32, 3] = 2.0 ** -25 * (1.0 + 2.0 ** -23)
    g = GaussianProcess(train, matern_nu=2.5, ell=[1.0] * 3, norm_offset=[0.0] * 3, norm_scale=[1.0] * 3, standard_mean=0.0,
                        standard_std=1.0, mean=0.0, sigma2=1.0, side=[10.0] * 3, precision=PGB_MIXED)
    want = 1.0 + train[32, 3] + (chunks - 2) * 2.0 ** -50
    assert np.all(np.abs(g(np.zeros((count, 3))) - want) <= chunks * 2.0 ** -53)
