"""The mixed slice terms' last step, the columns' Kahan sums over the lanes, is
in FP64: the bits of one slice's sums of the kernel with 128 threads a slice and
FP64 block sums (pairs of floats over the lanes differ from it in the last
three places of the centroid term)."""
import numpy as np
import pytest

from test_mixed_blocks import _pair, _path

pytestmark = pytest.mark.gpu

NAMES = ("vint", "g2", "r1", "r2", "d1", "d2", "kin", "xch")
SLICE3 = {
    129: ["-0x1.0edf5f3537e00p+11", "0x1.a4f7c09a4d000p+23", "-0x1.4a6663b1c0000p+11", "-0x1.8bff044b4da00p+25",
          "0x1.fcca000314000p+10", "0x1.44e01a175b500p+23", "0x1.3011a55e60000p+4", "0x1.112bac3be2000p+3"],
    200: ["-0x1.2bc6ff1f810c0p+12", "0x1.311db65f20c00p+19", "0x1.747bd0b188000p+11", "0x1.9fafab3a7b000p+21",
          "0x1.1296399d30000p+9", "0x1.5f7a0f51c8268p+19", "0x1.bf303da980000p+4", "0x1.a618b6823c000p+3"],
}


@pytest.mark.parametrize("n", sorted(SLICE3))
def test_one_slice(pgb, n):
    cfg, L = _path(pgb, n, 8, n)
    a, _ = _pair(pgb, cfg, L, 8, n)
    t = a.slice_terms()
    assert [float(t[k][3]).hex() for k in NAMES] == SLICE3[n]
