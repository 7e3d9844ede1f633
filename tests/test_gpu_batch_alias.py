"""Batch members that bind one of their pressure grids as a coefficient: it changes
with every sweep, so they take single sweeps whatever their bucket's entry says, and
end as the plain kernel's single sweeps do."""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("pressure", [0, 1])
@pytest.mark.parametrize("slot", [12, 13])
def test_coefficient_that_is_a_pressure_grid(slot, pressure, mode):
    ps.PSInit()
    dims, steps, out = (70, 40, 33), 6, []
    nx, ny, nz = dims
    p, coef = U.himeno_inputs((nz, ny, nx), 16)
    entry = dict(impl=ps.IMPL_TMA, tile_x=64, tile_y=8, z_chunk=8, stages=6)
    ps.batch_tune_set(ps.HIMENO19, dims, t_depth=2, **entry)
    try:
        for batch in (True, False):
            gs = [ps.grid_new(ps.PS_FLOAT, dims) for _ in range(14)]
            for g, a in zip(gs, [p, p] + list(coef)):
                ps.PSGridCopyin(g, a)
            bound = list(gs)
            bound[slot] = gs[pressure]
            if batch:
                b = ps.Batch()
                b.add(ps.HIMENO19, bound, [0.8], steps)
                b.run(mode)
                assert b.layout(0)["units"] == steps  # one sweep per item
                b.free()
            else:
                d = ps.PSDomain3DNew(1, nx - 1, 1, ny - 1, 1, nz - 1)
                ps.set_impl(ps.IMPL_PLAIN)
                ps.PSStencilRun(ps.PSStencilMap(ps.HIMENO19, d, *bound, 0.8),
                                ps.PSStencilMap(ps.HIMENO19, d, bound[1], bound[0], *bound[2:], 0.8),
                                steps // 2)
                ps.set_impl(ps.IMPL_AUTO)
            out.append([ps.PSGridCopyout(g) for g in gs[:2]])
            for g in gs:
                ps.PSGridFree(g)
    finally:
        ps.set_impl(ps.IMPL_AUTO)
        ps.batch_tune_set(ps.HIMENO19, dims, t_depth=1, **entry)
    assert U.bits_equal(out[0][0], out[1][0]) and U.bits_equal(out[0][1], out[1][1])
