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


# The second grid comes with values of its own (its rim stays in every second
# sweep), the domain is the interior or a part of it, and the passes start from
# the first grid (even pairs) or from a copy of it (odd ones).
@pytest.mark.parametrize("shape,cut", [((9, 11, 67), 0), ((20, 70, 131), 0), ((30, 41, 140), 3)])
@pytest.mark.parametrize("pairs", [2, 3, 4, 5])
def test_grids_with_different_rims_equal_plain(shape, cut, pairs):
    ps.PSInit()
    p, coef = U.himeno_inputs(shape, 12)
    other = np.random.default_rng(5).random(shape, dtype=np.float32)
    nz, ny, nx = shape
    out = []
    for impl in (ps.IMPL_AUTO, ps.IMPL_PLAIN):
        gs = [ps.grid_new(ps.PS_FLOAT, (nx, ny, nz)) for _ in range(14)]
        for g, a in zip(gs, [p, other] + list(coef)):
            ps.PSGridCopyin(g, a)
        d = ps.PSDomain3DNew(1 + cut, nx - 1 - cut, 1, ny - 1 - cut, 1 + cut, nz - 1)
        ps.set_impl(impl)
        try:
            m1 = ps.PSStencilMap(ps.HIMENO19, d, *gs, 0.8)
            m2 = ps.PSStencilMap(ps.HIMENO19, d, gs[1], gs[0], *gs[2:], 0.8)
            ps.PSStencilRun(m1, m2, pairs)
            out.append([ps.PSGridCopyout(g) for g in gs[:2]])
        finally:
            ps.set_impl(ps.IMPL_AUTO)
            for g in gs:
                ps.PSGridFree(g)
    assert U.bits_equal(out[0][0], out[1][0]) and U.bits_equal(out[0][1], out[1][1])


def test_halos_are_refreshed_after_a_run():
    """Both grids' halos (filled for periodic reads before the run) are stale
    after it: a periodic read two cells away sees the new values."""
    ps.PSInit()
    shape = (12, 14, 66)
    nz, ny, nx = shape
    p, coef = U.himeno_inputs(shape, 13)
    st = ps.GenericStencil(3, [(ps.PS_FLOAT, (0, 1, 2))] * 2, 1, ps.PS_FLOAT,
                           [(ps.get(0, [-2, 0, 0], ps.BOUNDARY_PERIODIC), ps.const(1.0)),
                            (ps.get(0, [0, 2, 0], ps.BOUNDARY_PERIODIC), ps.const(1.0))])
    gs = [ps.grid_new(ps.PS_FLOAT, (nx, ny, nz)) for _ in range(15)]
    try:
        for g, a in zip(gs, [p, p] + list(coef)):
            ps.PSGridCopyin(g, a)
        whole = ps.PSDomain3DNew(0, nx, 0, ny, 0, nz)
        reads = [ps.PSStencilMap(st.kernel_id, whole, g, gs[14]) for g in gs[:2]]
        for m in reads:
            ps.PSStencilRun(m, 1)
        d = ps.PSDomain3DNew(1, nx - 1, 1, ny - 1, 1, nz - 1)
        ps.PSStencilRun(ps.PSStencilMap(ps.HIMENO19, d, *gs[:14], 0.8),
                        ps.PSStencilMap(ps.HIMENO19, d, gs[1], gs[0], *gs[2:14], 0.8), 4)
        for g, m in zip(gs[:2], reads):
            a = ps.PSGridCopyout(g)
            ps.PSStencilRun(m, 1)
            want = np.roll(a, 2, axis=2) + np.roll(a, -2, axis=1)
            assert U.bits_equal(ps.PSGridCopyout(gs[14]), want)
    finally:
        for g in gs:
            ps.PSGridFree(g)


# Slots of the coefficient (wrk1, bnd, the first field) that is one of the two
# pressure grids: it changes with every sweep, and each point reads its own
# before it is stored.
@pytest.mark.parametrize("slot", [12, 13, 2])
@pytest.mark.parametrize("pressure", [0, 1])
def test_coefficient_that_is_a_pressure_grid_equals_plain(slot, pressure):
    ps.PSInit()
    shape, pairs = (20, 30, 131), 4
    nz, ny, nx = shape
    p, coef = U.himeno_inputs(shape, 14)
    other = np.random.default_rng(6).random(shape, dtype=np.float32)
    out = []
    for impl in (ps.IMPL_AUTO, ps.IMPL_PLAIN):
        gs = [ps.grid_new(ps.PS_FLOAT, (nx, ny, nz)) for _ in range(14)]
        for g, a in zip(gs, [p, other] + list(coef)):
            ps.PSGridCopyin(g, a)
        bound = list(gs)
        bound[slot] = gs[pressure]
        d = ps.PSDomain3DNew(1, nx - 1, 1, ny - 1, 1, nz - 1)
        ps.set_impl(impl)
        try:
            m1 = ps.PSStencilMap(ps.HIMENO19, d, *bound, 0.8)
            m2 = ps.PSStencilMap(ps.HIMENO19, d, bound[1], bound[0], *bound[2:], 0.8)
            ps.PSStencilRun(m1, m2, pairs)
            assert ps.last_run_stats()[1] == 2 * pairs  # single sweeps
            out.append([ps.PSGridCopyout(g) for g in gs[:2]])
        finally:
            ps.set_impl(ps.IMPL_AUTO)
            for g in gs:
                ps.PSGridFree(g)
    assert U.bits_equal(out[0][0], out[1][0]) and U.bits_equal(out[0][1], out[1][1])
