"""The staged form of checked stencil functions against the function's own
form, over every kind of block it is compiled for: tiles inside the grid, at
x faces only, at y and z faces, partial vectors at a domain's ends, lanes and
rows outside the domain, thin grids without any inner block."""
import numpy as np
import pytest

import physis_b200 as ps
from physis_b200 import dsl
from physis_b200.workloads import DIFFUSION7_DSL
from tests import gpu_util as U

pytestmark = pytest.mark.gpu

# Reads two points away with only one side tested (the other leaves the grid
# and reads 0, which is reported), values that depend on the coordinates, and
# a second grid; float and double.
SOURCE = """
void wide(const int x, const int y, const int z, PSGrid3D%(T)s u, PSGrid3D%(T)s w,
          PSGrid3D%(T)s v, %(t)s c) {
  const int nx = PSGridDim(u, 0), nz = PSGridDim(w, 2);
  %(t)s s = PSGridGet(u, x, y, z) * c;
  s = s + (x < 2 ? c : PSGridGet(u, x - 2, y, z));
  s = s + (x == nx - 1 ? PSGridGet(w, x, y, z) : PSGridGet(u, x + 1, y, z));
  s = s + PSGridGet(u, x, y + 2, z);
  s = s + (z == nz - 1 ? c : PSGridGet(w, x, y, z + 1));
  s = s + (z < 1 ? c : PSGridGet(w, x, y - 1, z - 1));
  PSGridEmit(v, s + c * (x + 2 * y + 3 * z));
}
"""
SHAPES = [(5, 4, 3), (130, 40, 9), (300, 21, 13), (257, 70, 6), (520, 18, 20)]


def _both(kernel, dims, typ, dom, params, ngrids):
    outs, forms = [], []
    rng = np.random.default_rng(sum(dims))
    fields = [rng.random(dims[::-1]).astype(ps.NP_TYPE[typ]) for _ in range(ngrids)]
    for mode in (ps.IMPL_AUTO, ps.IMPL_GENERIC):
        gs = [ps.grid_new(typ, dims) for _ in range(ngrids)]
        try:
            for g, f in zip(gs, fields):
                ps.PSGridCopyin(g, f)
            ps.set_impl(mode)
            ps.PSStencilRun(ps.PSStencilMap(kernel, dom, *gs, *params), 1)
            try:
                ps.sync()
                err = 0
            except ps.PhysisError as e:
                err = e.status
            forms.append((ps.compiled_last_staged(), err))
            outs.append(ps.PSGridCopyout(gs[-1]))
        finally:
            ps.set_impl(ps.IMPL_AUTO)
            for g in gs:
                ps.PSGridFree(g)
    return outs, forms


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    ps.PSInit()
    cache = str(tmp_path_factory.mktemp("dsl"))
    out = {}
    for typ, T, t in ((ps.PS_FLOAT, "Float", "float"), (ps.PS_DOUBLE, "Double", "double")):
        out[typ] = dsl.compile_stencils(SOURCE % {"T": T, "t": t}, cache)["wide"].kernel_id
    out["diffusion"] = dsl.compile_stencils(DIFFUSION7_DSL, cache)["diffusion7"].kernel_id
    return out


@pytest.mark.parametrize("inset", [0, 1, 3])
@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("which", ["float", "double", "diffusion"])
def test_every_kind_of_block_equals_the_own_form(which, dims, inset, kernels):
    if min(dims) - 2 * inset <= 0:
        pytest.skip("no domain left")
    dom = ps.PSDomain3DNew(*[v for n in dims for v in (inset, n - inset)])
    if which == "diffusion":
        got = _both(kernels["diffusion"], dims, ps.PS_FLOAT, dom, [0.1] * 6 + [0.4], 2)
    else:
        typ = ps.PS_FLOAT if which == "float" else ps.PS_DOUBLE
        got = _both(kernels[typ], dims, typ, dom, [0.3], 3)
    (a, b), (staged, own) = got
    assert U.bits_equal(a, b)
    assert staged[0] in (1, 2) and own[0] == 0
    assert staged[1] == own[1]
