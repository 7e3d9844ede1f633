"""Passes of several 7-point steps (k_diff7_pipe) against single steps.

PSStencilRun(m(A->B), m(B->A), iter) over whole pitched grids runs passes of
two and four steps where they are estimated faster; both grids must end bit
for bit as after the same maps run one at a time (which never fuse): float
and double, clamped and periodic, exact and FMA arithmetic, extents that end
inside a vector, inside a thread's rows and at tile edges, one tile and many,
z chunks that end early, every remainder of the step count.
"""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu

COEF = [0.11, 0.09, 0.1, 0.12, 0.08, 0.1, 0.4]
# (nx, ny, nz): tiny; ragged; one vector row; several tiles in x (odd) and y;
# long z; wide and flat.
SHAPES = [(4, 4, 4), (5, 9, 33), (64, 64, 64), (67, 50, 41), (130, 97, 20), (253, 61, 9),
          (31, 200, 12), (32, 12, 150), (500, 33, 6)]


def _run(shape, dtype, periodic, iters, fused):
    """Both grids after `iters` pairs, and the launches of the run."""
    t = ps.PS_FLOAT if dtype == np.float32 else ps.PS_DOUBLE
    nx, ny, nz = shape
    f = np.random.default_rng(nx + ny + nz).random((nz, ny, nx)).astype(dtype)
    a, b = ps.grid_new(t, shape), ps.grid_new(t, shape)
    try:
        ps.PSGridCopyin(a, f)
        d = ps.PSDomain3DNew(0, nx, 0, ny, 0, nz)
        k = ps.DIFFUSION7_PERIODIC if periodic else ps.DIFFUSION7
        m1, m2 = ps.PSStencilMap(k, d, a, b, *COEF), ps.PSStencilMap(k, d, b, a, *COEF)
        if fused:
            ps.PSStencilRun(m1, m2, iters)
            launches = ps.last_run_stats()[1]
        else:
            launches = 2 * iters
            for _ in range(iters):
                ps.PSStencilRun(m1, 1)
                ps.PSStencilRun(m2, 1)
        return ps.PSGridCopyout(a), ps.PSGridCopyout(b), launches
    finally:
        ps.PSGridFree(a)
        ps.PSGridFree(b)


@pytest.mark.parametrize("fma", [False, True], ids=["exact", "fma"])
@pytest.mark.parametrize("periodic", [False, True], ids=["clamped", "periodic"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_passes_equal_single_steps(shape, dtype, periodic, fma):
    ps.PSInit()
    ps.set_fp_mode(ps.FP_FMA if fma else ps.FP_EXACT)
    try:
        for iters in (2, 3, 6, 9):
            got = _run(shape, dtype, periodic, iters, True)
            want = _run(shape, dtype, periodic, iters, False)
            assert U.bits_equal(got[0], want[0]), iters
            assert U.bits_equal(got[1], want[1]), iters
    finally:
        ps.set_fp_mode(ps.FP_EXACT)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_every_mix_of_passes(dtype):
    """Step counts whose plans mix passes of four, three and two steps."""
    ps.PSInit()
    shape = (130, 97, 64)
    for iters in (4, 5, 7, 8, 10):
        got = _run(shape, dtype, False, iters, True)
        want = _run(shape, dtype, False, iters, False)
        assert got[2] < 2 * iters
        assert U.bits_equal(got[0], want[0]) and U.bits_equal(got[1], want[1]), iters


def test_large_runs_are_fused():
    """At 128^3 a run of 40 steps runs passes (fewer launches than steps)."""
    ps.PSInit()
    for periodic in (False, True):
        assert _run((128, 128, 128), np.float32, periodic, 20, True)[2] < 40


@pytest.mark.parametrize("iters", [1, 4])
def test_periodic_table_after_periodic_steps_sees_the_whole_halo(iters):
    """7-point steps keep only part of the periodic halo current; a table
    that reads the corners afterwards must see the wrapped values."""
    ps.PSInit()
    n = 24
    f = np.random.default_rng(3).random((n, n, n))
    a, b, c = (ps.PSGrid3DDoubleNew(n, n, n) for _ in range(3))
    try:
        ps.PSGridCopyin(a, f)
        d = ps.PSDomain3DNew(0, n, 0, n, 0, n)
        m1 = ps.PSStencilMap(ps.DIFFUSION7_PERIODIC, d, a, b, *COEF)
        m2 = ps.PSStencilMap(ps.DIFFUSION7_PERIODIC, d, b, a, *COEF)
        ps.PSStencilRun(m1, m2, iters)
        u = ps.PSGridCopyout(a)
        ax = (0, 1, 2)
        st = ps.GenericStencil(3, [(ps.PS_DOUBLE, ax)] * 2, 1, ps.PS_DOUBLE,
                               [ps.get(0, (2, 2, 2), ps.BOUNDARY_PERIODIC),
                                ps.get(0, (-1, -2, -1), ps.BOUNDARY_PERIODIC)])
        ps.PSStencilRun(ps.PSStencilMap(st.kernel_id, d, a, c), 1)
        want = np.roll(u, (-2, -2, -2), ax) + np.roll(u, (1, 2, 1), ax)
        assert U.bits_equal(ps.PSGridCopyout(c), want)
    finally:
        for g in (a, b, c):
            ps.PSGridFree(g)
