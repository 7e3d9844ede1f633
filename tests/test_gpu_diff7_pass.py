"""Every depth of a 7-point pass (k_diff7_pipe) at every shape, whatever a run
would choose: psb_diff7_pass forces the steps of a pass, and its tile and z chunk
too. A pass from one grid to the other and one back must leave both grids bit for
bit as that many single steps do; the second one reads the halo that the first
left (periodic grids)."""
import ctypes

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
# Threads a block, log2 of the lanes a row, z chunk: the smallest tiles and
# chunks, chunks that end early, one chunk, the largest blocks.
TILES = {2: [None, (64, 3, 1), (96, 4, 5), (128, 5, 3), (192, 3, 1000)],
         3: [None, (64, 3, 1), (96, 4, 5), (160, 5, 3), (384, 4, 1000)],
         4: [None, (64, 3, 1), (96, 4, 5), (192, 5, 3), (384, 4, 1000)]}

_pass = ps.lib.psb_diff7_pass
_pass.restype = ctypes.c_int
_pass.argtypes = [ctypes.c_int] * 5


def _one_pass(m, steps, tile):
    ps.check(_pass(m.handle, steps, *(tile or (0, 0, 0))), "psb_diff7_pass")
    assert ps.last_run_stats()[1] == 1


@pytest.mark.parametrize("fma", [False, True], ids=["exact", "fma"])
@pytest.mark.parametrize("kernel,steps", [(ps.DIFFUSION7, 2), (ps.DIFFUSION7, 3),
                                          (ps.DIFFUSION7, 4), (ps.DIFFUSION7_PERIODIC, 2)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_pass_equals_single_steps(shape, dtype, kernel, steps, fma):
    ps.PSInit()
    t = ps.PS_FLOAT if dtype == np.float32 else ps.PS_DOUBLE
    nx, ny, nz = shape
    f = np.random.default_rng(nx + ny + nz).random((nz, ny, nx)).astype(dtype)
    d = ps.PSDomain3DNew(0, nx, 0, ny, 0, nz)
    gs = [ps.grid_new(t, shape) for _ in range(2)]
    ps.set_fp_mode(ps.FP_FMA if fma else ps.FP_EXACT)
    try:
        ms = [ps.PSStencilMap(kernel, d, gs[i], gs[1 - i], *COEF) for i in (0, 1)]
        ps.PSGridCopyin(gs[0], f)
        want = []
        for k in range(2 * steps):
            ps.PSStencilRun(ms[k & 1], 1)
            if (k + 1) % steps == 0:
                want.append(ps.PSGridCopyout(gs[1 - (k & 1)]))
        for tile in TILES[steps]:
            ps.PSGridCopyin(gs[0], f)
            ps.PSGridCopyin(gs[1], np.full_like(f, np.nan))
            _one_pass(ms[0], steps, tile)
            first = ps.PSGridCopyout(gs[1])
            _one_pass(ms[1], steps, tile)
            assert U.bits_equal(first, want[0]), tile
            assert U.bits_equal(ps.PSGridCopyout(gs[0]), want[1]), tile
            assert U.bits_equal(ps.PSGridCopyout(gs[1]), first), tile
    finally:
        ps.set_fp_mode(ps.FP_EXACT)
        for g in gs:
            ps.PSGridFree(g)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("follow", ["table", "step"])
def test_readers_after_a_periodic_pass_see_their_halo(dtype, follow):
    """A pass leaves the images that the next pass reads; a table that reads the
    corners and a single step, which reads the z faces too, must see theirs."""
    ps.PSInit()
    t = ps.PS_FLOAT if dtype == np.float32 else ps.PS_DOUBLE
    n = 24
    f = np.random.default_rng(3).random((n, n, n)).astype(dtype)
    a, b, c = (ps.grid_new(t, (n, n, n)) for _ in range(3))
    d = ps.PSDomain3DNew(0, n, 0, n, 0, n)
    try:
        ps.PSGridCopyin(a, f)
        _one_pass(ps.PSStencilMap(ps.DIFFUSION7_PERIODIC, d, a, b, *COEF), 2, None)
        u = ps.PSGridCopyout(b)
        if follow == "table":
            ax = (0, 1, 2)
            st = ps.GenericStencil(3, [(t, ax)] * 2, 1, t,
                                   [ps.get(0, (2, 2, 2), ps.BOUNDARY_PERIODIC),
                                    ps.get(0, (-1, -2, -1), ps.BOUNDARY_PERIODIC)])
            ps.PSStencilRun(ps.PSStencilMap(st.kernel_id, d, b, c), 1)
            want = np.roll(u, (-2, -2, -2), ax) + np.roll(u, (1, 2, 1), ax)
        else:
            ps.PSStencilRun(ps.PSStencilMap(ps.DIFFUSION7_PERIODIC, d, b, c, *COEF), 1)
            ps.PSGridCopyin(a, u)  # the same values, no halo
            got = ps.PSGridCopyout(c)
            ps.PSStencilRun(ps.PSStencilMap(ps.DIFFUSION7_PERIODIC, d, a, c, *COEF), 1)
            want, c2 = ps.PSGridCopyout(c), got
            assert U.bits_equal(c2, want)
        assert U.bits_equal(ps.PSGridCopyout(c), want)
    finally:
        for g in (a, b, c):
            ps.PSGridFree(g)


def test_maps_that_passes_do_not_apply_to_are_refused():
    ps.PSInit()
    a, b = ps.grid_new(ps.PS_FLOAT, (16, 16, 16)), ps.grid_new(ps.PS_FLOAT, (16, 16, 16))
    e, g = (ps.grid_new(ps.PS_FLOAT, (16, 16, 16), ps.LAYOUT_DENSE) for _ in range(2))
    try:
        whole, part = ps.PSDomain3DNew(*(0, 16) * 3), ps.PSDomain3DNew(1, 16, 0, 16, 0, 16)
        for m, steps in ((ps.PSStencilMap(ps.DIFFUSION7, part, a, b, *COEF), 2),
                         (ps.PSStencilMap(ps.DIFFUSION7, whole, e, g, *COEF), 2),
                         (ps.PSStencilMap(ps.DIFFUSION7_PERIODIC, whole, a, b, *COEF), 4),
                         (ps.PSStencilMap(ps.DIFFUSION7, whole, a, b, *COEF), 5)):
            assert _pass(m.handle, steps, 0, 0, 0) != 0
    finally:
        for x in (a, b, e, g):
            ps.PSGridFree(x)
