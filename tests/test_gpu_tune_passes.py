"""What a tune entry says about passes of several 7-point steps: t_depth 1, which
psb_tune_get reports for a shape without an entry, leaves them to the library
(so setting what was got changes nothing), 2 makes them passes of two steps, 0
and the plain kernel keep single steps; the same for every 7-point kind, and the
same bits each time."""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu

COEF = [0.11, 0.09, 0.1, 0.12, 0.08, 0.1, 0.4]


@pytest.mark.parametrize("kernel,dtype,dims,pairs", [
    (ps.DIFFUSION7, np.float32, (130, 97, 64), 8),
    (ps.DIFFUSION7, np.float64, (130, 97, 64), 8),
    (ps.DIFFUSION7_PERIODIC, np.float32, (128, 128, 128), 20)])
def test_entries_of_every_kind(kernel, dtype, dims, pairs):
    ps.PSInit()
    t = ps.PS_FLOAT if dtype == np.float32 else ps.PS_DOUBLE
    nx, ny, nz = dims
    f = np.random.default_rng(9).random((nz, ny, nx)).astype(dtype)
    a, b = ps.grid_new(t, dims), ps.grid_new(t, dims)
    d = ps.PSDomain3DNew(0, nx, 0, ny, 0, nz)
    m1, m2 = ps.PSStencilMap(kernel, d, a, b, *COEF), ps.PSStencilMap(kernel, d, b, a, *COEF)
    old = ps.tune_get(kernel, t, dims)

    def run(**entry):
        if entry:
            ps.tune_set(kernel, t, dims, **dict(old, **entry))
        ps.PSGridCopyin(a, f)
        ps.PSStencilRun(m1, m2, pairs)
        return ps.last_run_stats()[1], ps.PSGridCopyout(a), ps.PSGridCopyout(b)

    try:
        free = run()
        assert free[0] < 2 * pairs  # passes
        two = (pairs - 1) & ~1
        for entry, launches in (({"t_depth": old["t_depth"]}, free[0]), ({"t_depth": 0}, 2 * pairs),
                                ({"t_depth": 2}, two + 2 * (pairs - two)),
                                ({"impl": ps.IMPL_PLAIN}, 2 * pairs), ({"t_depth": 1}, free[0])):
            got = run(**entry)
            assert got[0] == launches, entry
            assert U.bits_equal(got[1], free[1]) and U.bits_equal(got[2], free[2]), entry
    finally:
        ps.tune_set(kernel, t, dims, **old)
        ps.PSGridFree(a)
        ps.PSGridFree(b)
