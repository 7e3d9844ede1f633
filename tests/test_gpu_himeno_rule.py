"""Himeno runs without a tune entry (two sweeps per pass, chunk by rule) and
the narrow single-sweep tiles, against the plain kernel: bit for bit, with
the residual of every sweep (its sum order differs: 1e-12 relative)."""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu


# Extents: smallest interior; one tile exactly and one past it; narrow tiles
# (32 x 16) with a remainder; z chunks of one item and many.
@pytest.mark.parametrize("shape", [(3, 3, 3), (9, 10, 66), (9, 11, 67), (40, 35, 98), (150, 9, 34),
                                   (20, 70, 131)])
@pytest.mark.parametrize("sweeps", [2, 4, 6, 12])
def test_run_without_an_entry_equals_plain(shape, sweeps):
    ps.PSInit()
    p, coef = U.himeno_inputs(shape, 11)
    got, gosa = U.himeno_gpu(p, coef, 0.8, sweeps)
    want, wgosa = U.himeno_gpu(p, coef, 0.8, sweeps, impl=ps.IMPL_PLAIN)
    assert U.bits_equal(got, want)
    assert np.allclose(gosa, wgosa, rtol=1e-12, atol=0)
