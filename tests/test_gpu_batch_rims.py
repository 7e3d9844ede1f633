"""Batch members whose two pressure grids hold different values around the domain:
two sweeps per item would take the input's for both sweeps, so such a member takes
single sweeps, and takes two again once the grids agree; both ways its result is
that of the plain kernel's single sweeps, and with single sweeps so is its other
grid."""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu

DIMS, STEPS = (70, 40, 33), 6


def _fill(gs, p, other, coef):
    for g, a in zip(gs, [p, other] + list(coef)):
        ps.PSGridCopyin(g, a)


def _plain(p, other, coef):
    nx, ny, nz = DIMS
    gs = [ps.grid_new(ps.PS_FLOAT, DIMS) for _ in range(14)]
    _fill(gs, p, other, coef)
    d = ps.PSDomain3DNew(1, nx - 1, 1, ny - 1, 1, nz - 1)
    ps.set_impl(ps.IMPL_PLAIN)
    try:
        ps.PSStencilRun(ps.PSStencilMap(ps.HIMENO19, d, *gs, 0.8),
                        ps.PSStencilMap(ps.HIMENO19, d, gs[1], gs[0], *gs[2:], 0.8), STEPS // 2)
    finally:
        ps.set_impl(ps.IMPL_AUTO)
    out = [ps.PSGridCopyout(g) for g in gs[:2]]
    for g in gs:
        ps.PSGridFree(g)
    return out


@pytest.mark.parametrize("mode", [0, 1])
def test_members_with_different_rims(mode):
    ps.PSInit()
    p, coef = U.himeno_inputs(DIMS[::-1], 17)
    corner, face = p.copy(), p.copy()
    corner[-1, -1, -1] += 0.5       # the one cell that no point of the domain reads
    face[5, 7, -1] -= 0.25          # one that two sweeps read
    entry = dict(impl=ps.IMPL_TMA, tile_x=64, tile_y=8, z_chunk=8, stages=6)
    ps.batch_tune_set(ps.HIMENO19, DIMS, t_depth=2, **entry)
    gs = [ps.grid_new(ps.PS_FLOAT, DIMS) for _ in range(14)]
    b = ps.Batch()
    try:
        b.add(ps.HIMENO19, gs, [0.8], STEPS)
        for other, units in ((p, STEPS // 2), (face, STEPS), (face, STEPS), (p, STEPS // 2),
                             (corner, STEPS)):
            _fill(gs, p, other, coef)
            b.run(mode)
            assert b.layout(0)["units"] == units
            want = _plain(p, other, coef)
            done, _, g = b.result(0)
            assert done == STEPS
            assert U.bits_equal(ps.PSGridCopyout(g), want[0])
            if units == STEPS:
                assert U.bits_equal(ps.PSGridCopyout(gs[1]), want[1])
    finally:
        b.free()
        ps.batch_tune_set(ps.HIMENO19, DIMS, t_depth=1, **entry)
        for g in gs:
            ps.PSGridFree(g)
