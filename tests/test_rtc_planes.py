"""The plane-by-plane kernel body (gt_body_planes) and the point kernel's
helpers (k_generic_pt.cuh) compile under NVRTC without host headers, in
programs of the shape the library generates at run time (CPU only; see
test_rtc_headers.py for the window form)."""
import pytest

from tests.test_rtc_headers import CSRC, _compile, nvrtc

# Two grids, a window of three planes, shared and unit coefficients.
PLANES = r"""
#include "k_generic_tma.cuh"
namespace psb {
struct GtPlaneProg {
  static constexpr int kWindow = 3;
  template <typename T>
  static __device__ __forceinline__ void plane(const GtTable &tab, const T *p, int bx,
      int plane_elems, int lane, GtBlk<T> *acc) {
    GtRow<T> q0[kGtVY + 2 * kGtR];
    gt_row_ext<T, false, true, true, false>(p + 0 * plane_elems + (-1) * bx, lane, q0[1]);
    gt_row_ext<T, true, true, true, true>(p + 0 * plane_elems + (0) * bx, lane, q0[2]);
    gt_row_ext<T, false, false, false, false>(p + 0 * plane_elems + (1) * bx, lane, q0[3]);
    gt_row_ext<T, false, false, false, false>(p + 0 * plane_elems + (2) * bx, lane, q0[4]);
    gt_row_ext<T, false, false, false, false>(p + 0 * plane_elems + (3) * bx, lane, q0[5]);
    GtRow<T> q1[kGtVY + 2 * kGtR];
    for (int y = 0; y < 4; y++)
      gt_row_ext<T, false, false, false, false>(p + 1 * plane_elems + y * bx, lane, q1[2 + y]);
    const T c0 = gt_coef(tab, 0, T());
    (void)c0;
    gt_plane_term<T, -1, 1, false, true, FMA>(q0, c0, acc[0]);
    gt_plane_term<T, 0, 4, true, false, FMA>(q0, c0, acc[2]);
    gt_plane_term<T, 0, 2, false, false, FMA>(q1, c0, acc[1]);
  }
};
}  // namespace psb
extern "C" __global__ void __launch_bounds__(psb::kGtThreads, 3)
psb_generic_tma_compiled(const __grid_constant__ psb::GtMaps maps,
                         const __grid_constant__ psb::GtTable tab, psb::GridView out,
                         psb::Dom3 d, const __grid_constant__ psb::GtGeom geo, int *err) {
  psb::gt_body_planes<TYPE, psb::GtPlaneProg>(maps, tab, out, d, geo, err);
}
"""

# A red-black point: periodic, clamped and plain indices, mixed types.
POINTS = r"""
#include "k_generic_pt.cuh"
extern "C" __global__ void __launch_bounds__(256) psb_generic_points(
    const __grid_constant__ psb::GpArgs q) {
  using namespace psb;
  typedef double A;
  const float *const g0 = (const float *)q.g[0].origin;
  const int64_t *const g1 = (const int64_t *)q.g[1].origin;
  const int64_t sy0 = q.g[0].sy;
  const GpAt at = gp_position<2, 4, true>(q);
  const int x = at.x, y = at.y, px = at.px;
  if (x + px >= q.d.hi[0] || y >= q.d.hi[1]) return;
  A v = (A)gp_ld<false>(g0 + (int64_t)gp_wrap(x + px - 1, q.g[0].n[0]) + (int64_t)y * sy0);
  v = xadd(v, xmul((A)gp_ld<true>(g1 + gp_clamp(x - 2, q.g[1].n[0])), (A)q.b[0]));
  v = xmul(v, (A)gp_ld<true>(g1 + gp_mod(x + 9, q.g[1].n[0])));
  *const_cast<float *>(g0 + x + (int64_t)y * sy0) = (float)v;
}
"""


def _opts():
    return ["--gpu-architecture=sm_100a", "-std=c++17", "--fmad=false", "-default-device",
            "-I" + CSRC]


@pytest.mark.parametrize("typ", ["float", "double"])
@pytest.mark.parametrize("fma", ["true", "false"])
def test_plane_form_compiles(typ, fma):
    src = PLANES.replace("TYPE", typ).replace("FMA", fma)
    res, log, size = _compile(src, _opts() + ["-DPSB_GT_VY=4"])
    assert res == nvrtc.nvrtcResult.NVRTC_SUCCESS, log
    assert size > 0


def test_point_kernel_compiles():
    res, log, size = _compile(POINTS, _opts())
    assert res == nvrtc.nvrtcResult.NVRTC_SUCCESS, log
    assert size > 0
