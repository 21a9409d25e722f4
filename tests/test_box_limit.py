"""A box whose potential table would not fit 31-bit indexes is refused before
any device memory is touched."""
import numpy as np
import pytest


@pytest.mark.parametrize("side", [8000.0, [27000.0, 24000.0, 7.0], [1e9, 5.0, 5.0], [np.nan, 9.0, 9.0], [np.inf, 9.0, 9.0]])
def test_refused(pgb, side):
    with pytest.raises(pgb.PgbError) as e:
        pgb.Action(side, 4, 4, 0.004, 6.0596)
    assert e.value.code == -1 and "table" in str(e.value)
