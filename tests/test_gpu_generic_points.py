"""Generic stencils outside the TMA path: the kernel compiled for the table
against the kernel that interprets it (bit for bit).

Random tables over ranks, element types, index forms (with offsets beyond one
period), grids of lower dimension, red-black passes, in-place updates,
sub-domains and both layouts, at sizes on both sides of the line between one
and four points a thread, with extents that leave partial blocks, partial
groups of four and odd column pairs.
"""
import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U

pytestmark = pytest.mark.gpu

TYPES = [ps.PS_INT, ps.PS_LONG, ps.PS_FLOAT, ps.PS_DOUBLE]
# Extents: tiny, one point a thread, four points a thread (the last of each
# rank; coloured passes have half the points).
SHAPES = {1: [(3,), (1025,), (700001,)], 2: [(5, 3), (129, 66), (1203, 1101)],
          3: [(5, 4, 3), (33, 17, 30), (131, 126, 79)]}


def _factor(rng, slot, nd, axes, lo, hi, dims, inplace):
    if slot is None:
        return ps.const(float(rng.choice([1.0, -2.0, 3.0])))
    if inplace:
        return ps.get(slot)
    b = int(rng.integers(0, 3))
    off = [0, 0, 0]
    for k in range(nd):
        off[k] = int(rng.integers(-2, 3)) if rng.random() < 0.9 or b == 0 else int(dims[k]) + 1
        if b == 0:  # plain reads stay inside the grid
            off[k] = min(max(off[k], -lo[k]), dims[k] - hi[k])
        elif b == 1:  # (i + n) % n is an index for offsets down to -n
            off[k] = min(max(off[k], -dims[k]), dims[k] + 1)
    return ps.get(slot, off, b)


def _case(seed, nd, size, colored):
    rng = np.random.default_rng(1000 * seed + 10 * nd + size + (5 if colored else 0))
    dims = SHAPES[nd][size]
    lo = [int(rng.integers(0, 2)) for _ in dims]
    hi = [int(n - rng.integers(0, 2)) for n in dims]
    accum = TYPES[int(rng.integers(0, 4))]
    grids, out = [], int(rng.integers(0, 3))
    for i in range(3):
        axes = tuple(range(nd))
        if i != out and nd > 1 and rng.random() < 0.4:
            axes = tuple(sorted(rng.choice(nd, int(rng.integers(1, nd)), replace=False).tolist()))
        grids.append((TYPES[int(rng.integers(0, 4))], axes))
    pick = lambda: int(rng.integers(0, 3)) if rng.random() < 0.8 else None  # noqa: E731

    def factor():
        s = pick()
        return _factor(rng, s, nd, None if s is None else grids[s][1], lo, hi, dims, s == out)

    terms = [(factor(), factor()) for _ in range(int(rng.integers(1, 8)))]
    post = factor() if rng.random() < 0.5 else None
    values = []
    for t, axes in grids:
        shape = tuple(dims[a] for a in reversed(axes))
        v = rng.integers(-3, 4, size=shape)
        values.append((v * (0.3 if t in (ps.PS_FLOAT, ps.PS_DOUBLE) else 1)).astype(ps.NP_TYPE[t]))
    return dict(ndims=nd, grids=grids, out=out, accum=accum, terms=terms, post=post), values, lo, hi


@pytest.mark.parametrize("layout", sorted(U.LAYOUTS))
@pytest.mark.parametrize("colored", [False, True], ids=["all", "redblack"])
@pytest.mark.parametrize("size", [0, 1, 2])
@pytest.mark.parametrize("nd", [1, 2, 3])
def test_compiled_points_equal_interpreted(nd, size, colored, layout):
    ps.PSInit()
    for seed in range(3):
        d, values, lo, hi = _case(seed, nd, size, colored)
        st = ps.GenericStencil(d["ndims"], d["grids"], d["out"], d["accum"], d["terms"], d["post"])
        dom = [ps.PSDomain1DNew, ps.PSDomain2DNew, ps.PSDomain3DNew][nd - 1](
            *[v for p in zip(lo, hi) for v in p])
        outs = []
        for mode in (ps.IMPL_AUTO, ps.IMPL_GENERIC):
            gs = [ps.grid_new(t, v.shape[::-1], U.LAYOUTS[layout])
                  for (t, _), v in zip(d["grids"], values)]
            try:
                for g, v in zip(gs, values):
                    ps.PSGridCopyin(g, v)
                ps.set_impl(mode)
                m = (ps.PSStencilMapRedBlack if colored else ps.PSStencilMap)(st.kernel_id, dom, *gs)
                ps.PSStencilRun(m, 1)
                outs.append(ps.PSGridCopyout(gs[d["out"]]))
            finally:
                ps.set_impl(ps.IMPL_AUTO)
                for g in gs:
                    ps.PSGridFree(g)
        assert U.bits_equal(outs[0], outs[1]), (seed, d)


def test_rows_of_a_red_black_pass_replayed_from_a_graph():
    """An in-place red-black relaxation of several iterations (the graph
    replays the compiled kernel) equals the interpreting kernel's."""
    ps.PSInit()
    nx, ny, nz = 67, 35, 41
    c = float(np.float32(1.0 / 6.0))
    terms = [(ps.const(c), ps.get(0, o)) for o in
             ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))]
    st = ps.GenericStencil(3, [(ps.PS_FLOAT, (0, 1, 2))], 0, ps.PS_FLOAT, terms)
    f = np.random.default_rng(4).random((nz, ny, nx), dtype=np.float32)
    outs = []
    for mode in (ps.IMPL_AUTO, ps.IMPL_GENERIC):
        g = ps.PSGrid3DFloatNew(nx, ny, nz)
        try:
            ps.PSGridCopyin(g, f)
            ps.set_impl(mode)
            m = ps.PSStencilMapRedBlack(st.kernel_id,
                                        ps.PSDomain3DNew(1, nx - 1, 1, ny - 1, 1, nz - 1), g)
            ps.PSStencilRun(m, 9)
            outs.append(ps.PSGridCopyout(g))
        finally:
            ps.set_impl(ps.IMPL_AUTO)
            ps.PSGridFree(g)
    assert U.bits_equal(outs[0], outs[1])
