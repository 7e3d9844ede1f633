"""Two maps that swap two grids run in passes of several steps only when their
scalars are the same numbers: 0 and -0 are not (they give zeros of other signs)."""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [ps.DIFFUSION7, ps.DIFFUSION7_PERIODIC])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_zero_and_minus_zero_coefficients(kernel, dtype):
    ps.PSInit()
    n, pairs = 128, 8
    t = ps.PS_FLOAT if dtype == np.float32 else ps.PS_DOUBLE
    f = np.full((n, n, n), -0.0, dtype)
    d = ps.PSDomain3DNew(0, n, 0, n, 0, n)
    out = []
    for together in (True, False):
        a, b = ps.grid_new(t, (n, n, n)), ps.grid_new(t, (n, n, n))
        ps.PSGridCopyin(a, f)
        m1 = ps.PSStencilMap(kernel, d, a, b, *[0.0] * 7)
        m2 = ps.PSStencilMap(kernel, d, b, a, *[-0.0] * 7)
        if together:
            ps.PSStencilRun(m1, m2, pairs)
        else:
            for _ in range(pairs):
                ps.PSStencilRun(m1, 1)
                ps.PSStencilRun(m2, 1)
        out.append((ps.PSGridCopyout(a), ps.PSGridCopyout(b)))
        ps.PSGridFree(a)
        ps.PSGridFree(b)
    # From -0 one pair gives -0 (0 * -0) and then 0 (-0 * -0), from 0 the next one 0 and -0.
    assert np.signbit(out[1][0]).all() and not np.signbit(out[1][1]).any()
    assert U.bits_equal(out[0][0], out[1][0]) and U.bits_equal(out[0][1], out[1][1])


def test_zero_and_minus_zero_relaxation():
    ps.PSInit()
    shape, pairs = (20, 30, 66), 3
    nz, ny, nx = shape
    p, coef = U.himeno_inputs(shape, 15)
    out = []
    for impl in (ps.IMPL_AUTO, ps.IMPL_PLAIN):
        gs = [ps.grid_new(ps.PS_FLOAT, (nx, ny, nz)) for _ in range(14)]
        for g, a in zip(gs, [np.full(shape, -0.0, np.float32)] * 2 + list(coef)):
            ps.PSGridCopyin(g, a)
        d = ps.PSDomain3DNew(1, nx - 1, 1, ny - 1, 1, nz - 1)
        ps.set_impl(impl)
        try:
            m1 = ps.PSStencilMap(ps.HIMENO19, d, *gs, -0.0)
            m2 = ps.PSStencilMap(ps.HIMENO19, d, gs[1], gs[0], *gs[2:], 0.0)
            ps.PSStencilRun(m1, m2, pairs)
            out.append([ps.PSGridCopyout(g) for g in gs[:2]])
        finally:
            ps.set_impl(ps.IMPL_AUTO)
            for g in gs:
                ps.PSGridFree(g)
    assert U.bits_equal(out[0][0], out[1][0]) and U.bits_equal(out[0][1], out[1][1])
