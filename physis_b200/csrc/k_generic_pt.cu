// Generic stencils outside the TMA path, compiled for their table.
//
// The reference's translator emits one kernel per stencil function
// (translator/cuda_translator.cc:615-869). A registered psb_generic_stencil
// that the plane pipeline (k_generic_tma.cu) does not take -- red-black
// order, in-place updates, one- and two-dimensional domains, mixed element
// types, grids of lower dimension, integer grids, offsets beyond the halo --
// is compiled here when its map runs (generic_note_uses says from when on): the
// term program is written out as straight-line code over the map's strided views, with every factor's
// grid, type, axes, offset and index form a constant.
//
// What bounds it: k_generic (k_generic.cu), which interprets the table,
// issues a few hundred instructions per term and point (the factor's record,
// its grid's view and type switch, 64-bit index arithmetic). Straight-line
// code leaves one load, one multiply and one add per term, so these maps are
// bound by L1/L2 traffic. A thread owns U consecutive planes (3-D) or rows
// (2-D): the loads that its points share along that axis are issued once,
// and the index arithmetic is paid once per thread. In a red-black pass the
// threads cover only the points of the pass's colour. Measured (float): a
// red-black iteration of a 7-term relaxation with a right-hand side at 256^3
// 68 us against 1624 us interpreted; a 5-point step at 4001 x 2003 11.0 us
// against 235 us.
//
// Arithmetic and order are those of k_generic, so results are bit-identical
// (a factor that is the constant 1 is not multiplied: x * 1 == x).
#include <algorithm>
#include <climits>
#include <cstring>
#include <string>

#include "internal.h"
#include "k_generic_pt.cuh"

namespace psb {
namespace {

// b / d as (b * mul) >> shift, exact for 0 <= b < 2^31: with 2^(l-1) < d <= 2^l
// and mul = floor(2^(31+l) / d) + 1, b * mul / 2^(31+l) exceeds b / d by less
// than 1 / d. (The divisions were 12 of 43 instructions a point: a 5-point step
// at 4001 x 2003 took 15.4 us with them.)
void gp_divisor(int d, unsigned *mul, int *shift) {
  int l = 0;
  while ((1ll << l) < d) l++;
  *shift = 31 + l;
  *mul = (unsigned)((1ull << *shift) / (unsigned)d + (d > 1));
}

const char *ctype(int t) {
  switch (t) {
    case PS_FLOAT: return "float";
    case PS_DOUBLE: return "double";
    case PS_INT: return "int32_t";
    default: return "int64_t";
  }
}

struct GpShape {
  bool colored;
  int U;
  bool nc[PSB_MAX_GRIDS];          // the slot's grid is not the written one
  bool one_period[PSB_MAX_GRIDS];  // periodic indices leave [0, n) by at most one period
};

std::string num(int v) { return "(" + std::to_string(v) + ")"; }

// The value of factor f (term t, side 'a' or 'b'; 'p' for the post factor)
// at the thread's point r, converted to A.
std::string factor_src(const psb_generic_stencil &d, const GpShape &sh, const psb_factor &f,
                       const std::string &side, int t, int r) {
  if (f.grid < 0) {
    const std::string arr = side + (d.accum_type == PS_FLOAT ? "32" : "");
    if (side == "post") return "(A)q." + arr;
    return "(A)q." + arr + "[" + std::to_string(t) + "]";
  }
  const int gi = f.grid;
  const std::string g = std::to_string(gi);
  std::string addr;
  const char *pos[3] = {"x", "y", "z"}, *stride[3] = {"1", "sy", "sz"};
  for (int k = 0; k < 3 && d.grid_axes[gi][k] >= 0; k++) {
    const int ax = d.grid_axes[gi][k];
    const int off = f.offset[ax];
    const bool walks = ax == d.ndims - 1 && ax > 0;  // the axis of the U points
    const std::string st = k == 0 ? "" : std::string(" * ") + stride[k] + g;
    std::string p = pos[ax];
    if (ax == 0 && sh.colored) p = (r & 1) ? "(x + (px ^ 1))" : "(x + px)";
    if (f.boundary == PSB_BOUNDARY_NONE) {
      // Base of the thread plus a constant number of strides.
      addr += " + (int64_t)" + p + st;
      const int c = off + (walks ? r : 0);
      if (c) addr += " + (int64_t)" + num(c) + st;
    } else {
      std::string i = p + " + " + num(off + (walks ? r : 0));
      if (!(off == 0 && sh.one_period[gi])) {
        const char *fn = f.boundary == PSB_BOUNDARY_CLAMP ? "gp_clamp"
                         : sh.one_period[gi]              ? "gp_wrap"
                                                          : "gp_mod";
        i = std::string(fn) + "(" + i + ", q.g[" + g + "].n[" + std::to_string(k) + "])";
      }
      addr += " + (int64_t)(" + i + ")" + st;
    }
  }
  return std::string("(A)gp_ld<") + (sh.nc[gi] ? "true" : "false") + ">(g" + g + addr + ")";
}

// Statements that leave the stencil's value at point r in v<r>.
std::string point_src(const psb_generic_stencil &d, const GpShape &sh, int r) {
  const std::string v = "v" + std::to_string(r);
  auto one = [](const psb_factor &f) { return f.grid < 0 && f.constant == 1.0; };
  std::string s;
  for (int t = 0; t < d.nterms; t++) {
    const psb_factor &a = d.terms[t].a, &b = d.terms[t].b;
    std::string e;
    if (one(b)) e = factor_src(d, sh, a, "a", t, r);
    else if (one(a)) e = factor_src(d, sh, b, "b", t, r);
    else e = "xmul(" + factor_src(d, sh, a, "a", t, r) + ", " + factor_src(d, sh, b, "b", t, r) + ")";
    s += "      " + v + " = " + (t ? "xadd(" + v + ", " + e + ")" : e) + ";\n";
  }
  if (d.has_post && !one(d.post))
    s += "      " + v + " = xmul(" + v + ", " + factor_src(d, sh, d.post, "post", 0, r) + ");\n";
  return s;
}

std::string store_src(const psb_generic_stencil &d, const GpShape &sh, int r) {
  const std::string o = std::to_string(d.out_grid);
  std::string addr = "g" + o + " + (int64_t)" +
                     (sh.colored ? ((r & 1) ? "(x + (px ^ 1))" : "(x + px)") : "x");
  if (d.ndims > 1)
    addr += " + (int64_t)y * sy" + o +
            (d.ndims == 2 && r ? " + (int64_t)" + num(r) + " * sy" + o : "");
  if (d.ndims > 2)
    addr += " + (int64_t)z * sz" + o + (r ? " + (int64_t)" + num(r) + " * sz" + o : "");
  return "      *const_cast<" + std::string(ctype(d.grid_type[d.out_grid])) + " *>(" + addr +
         ") = (" + ctype(d.grid_type[d.out_grid]) + ")v" + std::to_string(r) + ";\n";
}

std::string source_of(const psb_generic_stencil &d, const GpShape &sh) {
  // Short float tables run in 32 registers, eight blocks an SM: these maps wait
  // for memory (red-black 256^3: 770 us with the 39 the compiler takes, 683 with 32).
  bool slim = d.nterms <= 8 && d.accum_type == PS_FLOAT;
  for (int i = 0; i < d.ngrids; i++) slim = slim && d.grid_type[i] == PS_FLOAT;
  std::string s = std::string("#include \"k_generic_pt.cuh\"\n"
                              "static_assert(sizeof(psb::GpArgs) == " +
                              std::to_string(sizeof(GpArgs)) + ", \"as the host fills it\");\n"
                              "extern \"C\" __global__ void __launch_bounds__(256") +
                  (slim ? ", 8" : "") + ") "
                  "psb_generic_points(const __grid_constant__ psb::GpArgs q) {\n"
                  "  using namespace psb;\n  typedef " + std::string(ctype(d.accum_type)) + " A;\n";
  for (int i = 0; i < d.ngrids; i++) {
    const std::string g = std::to_string(i), T = ctype(d.grid_type[i]);
    s += "  const " + T + " *const g" + g + " = (const " + T + " *)q.g[" + g + "].origin;\n" +
         "  const int64_t sy" + g + " = q.g[" + g + "].sy, sz" + g + " = q.g[" + g + "].sz;\n" +
         "  (void)g" + g + "; (void)sy" + g + "; (void)sz" + g + ";\n";
  }
  const std::string U = std::to_string(sh.U);
  s += "  const GpAt at = gp_position<" + std::to_string(d.ndims) + ", " + U + ", " +
       (sh.colored ? "true" : "false") + ">(q);\n"
       "  const int x = at.x, y = at.y, z = at.z, px = at.px;\n  (void)px;\n"
       "  const int hx = q.d.hi[0], hy = q.d.hi[1], hz = q.d.hi[2];\n"
       "  if (x >= hx || y >= hy || z >= hz) return;\n";
  const char *walk = d.ndims == 3 ? "z" : d.ndims == 2 ? "y" : "x";
  // All U points inside: loads shared, stores last.
  if (sh.U > 1) {
    s += "  if (" + std::string(walk) + " + " + std::to_string(sh.U - 1) + " < h" + walk +
         (sh.colored ? " && x + 1 < hx" : "") + ") {\n    A ";
    for (int r = 0; r < sh.U; r++) s += (r ? ", v" : "v") + std::to_string(r);
    s += ";\n";
    for (int r = 0; r < sh.U; r++) s += point_src(d, sh, r);
    for (int r = 0; r < sh.U; r++) s += store_src(d, sh, r);
    s += "    return;\n  }\n";
  }
  for (int r = 0; r < sh.U; r++) {
    std::string in = std::string(walk) + " + " + std::to_string(r) + " < h" + walk;
    if (sh.colored) in += std::string(" && x + ") + ((r & 1) ? "(px ^ 1)" : "px") + " < hx";
    s += "  if (" + in + ") {\n    A v" + std::to_string(r) + ";\n" + point_src(d, sh, r) +
         store_src(d, sh, r) + "  }\n";
  }
  return s + "}\n";
}

std::string factor_key(const psb_generic_stencil &d, const psb_factor &f) {
  if (f.grid < 0) return f.constant == 1.0 ? "1" : "c";
  return std::to_string(f.grid) + "." + std::to_string(f.offset[0]) + "." +
         std::to_string(f.offset[1]) + "." + std::to_string(f.offset[2]) + "." +
         std::to_string(f.boundary);
}

std::string key_of(const psb_generic_stencil &d, const GpShape &sh) {
  std::string k = "k_generic_pt:" + std::to_string(d.ndims) + ":" + std::to_string(d.accum_type) +
                  ":" + std::to_string(d.out_grid) + ":" + std::to_string(sh.U) +
                  (sh.colored ? "c" : "a") + ":";
  for (int i = 0; i < d.ngrids; i++) {
    k += std::to_string(d.grid_type[i]) + (sh.one_period[i] ? "w" : "m") + (sh.nc[i] ? "n" : "p");
    for (int j = 0; j < 3; j++) k += "." + std::to_string(d.grid_axes[i][j]);
    k += ",";
  }
  for (int t = 0; t < d.nterms; t++)
    k += factor_key(d, d.terms[t].a) + "*" + factor_key(d, d.terms[t].b) + ",";
  if (d.has_post) k += "p" + factor_key(d, d.post);
  return k;
}

}  // namespace

// The compiler takes 40 ms (four terms, one point a thread) to 540 ms (32 terms,
// four points a thread: about 40 + 15 a term), interpreting 5 us an application
// and 14 ps a term and point: a table that is applied a few times is interpreted.
// It is compiled for the run that brings it to eight applications (a loop; each
// gains 2.4 to 15 times, from 16^3 up) or to as long as the compiler takes.
void generic_note_uses(GenericDesc &gd, double uses, double points) {
  gd.uses += uses;
  gd.work += uses * points * gd.host.nterms;
  gd.interpret =
      !generic_compile_forced() && gd.uses < 8 && gd.work < 1e9 * (3 + gd.host.nterms);
}

// PSB_ERR_UNSUPPORTED when the map keeps k_generic: a written grid that does
// not follow the domain's axes one to one, columns near the largest int, no
// run-time compiler, or a kernel that is not compiled yet while the table has
// been used too little or the stream is being captured.
psb_status generic_points_launch(MapImpl &m, const GenericDesc &gd, int color, cudaStream_t s,
                                 int64_t *launches) {
  const psb_generic_stencil &d = gd.host;
  if (!generic_compile_on()) return PSB_ERR_UNSUPPORTED;
  // The last block's columns past the domain must be ints too (a check in the
  // kernel costs every point of a short table).
  if (m.dom.local_max[0] > INT_MAX - 2 * kGpThreads) return PSB_ERR_UNSUPPORTED;
  for (int k = 0; k < 3; k++)
    if (d.grid_axes[d.out_grid][k] != (k < d.ndims ? k : -1)) return PSB_ERR_UNSUPPORTED;
  for (int i = 0; i < d.ngrids; i++)  // axes listed from the first, without gaps
    for (int k = 1; k < 3; k++)
      if (d.grid_axes[i][k] >= 0 && d.grid_axes[i][k - 1] < 0) return PSB_ERR_UNSUPPORTED;
  GpArgs q;
  memset(&q, 0, sizeof(q));
  int64_t ext[3];
  for (int i = 0; i < 3; i++) {
    q.d.lo[i] = i < d.ndims ? m.dom.local_min[i] : 0;
    q.d.hi[i] = i < d.ndims ? m.dom.local_max[i] : 1;
    ext[i] = (int64_t)q.d.hi[i] - q.d.lo[i];
  }
  q.color = color;
  GpShape sh;
  sh.colored = color >= 0;
  for (int i = 0; i < d.ngrids; i++) {
    q.g[i] = m.grids[i]->view();
    q.g[i].type = d.grid_type[i];
    sh.one_period[i] = true;
    sh.nc[i] = m.grids[i] != m.grids[d.out_grid];
    for (int k = 0; k < 3 && d.grid_axes[i][k] >= 0; k++) {
      const int ax = d.grid_axes[i][k];
      if (q.d.lo[ax] < 0 || q.d.hi[ax] > q.g[i].n[k]) sh.one_period[i] = false;
    }
  }
  auto take = [&](const psb_factor &f, double *c, float *c32) {
    if (f.grid < 0) {
      *c = f.constant;
      *c32 = (float)f.constant;
      return;
    }
    for (int k = 0; k < 3 && d.grid_axes[f.grid][k] >= 0; k++) {
      const int off = f.offset[d.grid_axes[f.grid][k]];
      if (off > q.g[f.grid].n[k] || off < -q.g[f.grid].n[k]) sh.one_period[f.grid] = false;
    }
  };
  for (int t = 0; t < d.nterms; t++) {
    take(d.terms[t].a, &q.a[t], &q.a32[t]);
    take(d.terms[t].b, &q.b[t], &q.b32[t]);
  }
  if (d.has_post) take(d.post, &q.post, &q.post32);
  // Four points a thread share loads along the walked axis once the grid
  // gives every SM a few blocks of them; smaller grids keep one point a
  // thread, where filling the SMs counts for more.
  const int64_t points = ext[0] * ext[1] * ext[2] / (sh.colored ? 2 : 1);
  sh.U = d.ndims > 1 && points >= (int64_t)rt().sm_count * 4 * kGpThreads * 4 ? 4 : 1;
  const int64_t slots = sh.colored ? (ext[0] + 1) / 2 : ext[0];
  if (d.ndims == 1) {
    q.tx_shift = 8;
  } else {
    q.tx_shift = 5;
    while (q.tx_shift > 2 && slots <= (1 << (q.tx_shift - 1))) q.tx_shift--;
  }
  const int64_t tx = 1 << q.tx_shift, ty = (kGpThreads / tx) * (d.ndims == 2 ? sh.U : 1);
  const int64_t tz = d.ndims == 3 ? sh.U : 1;
  const int64_t bx = (slots + tx - 1) / tx, by = (ext[1] + ty - 1) / ty, bz = (ext[2] + tz - 1) / tz;
  if (bx * by * bz > 0x7fffffff) return PSB_ERR_UNSUPPORTED;
  q.tiles_x = (int)bx;
  q.tiles_y = (int)by;
  gp_divisor(q.tiles_x, &q.mul_x, &q.shift_x);
  gp_divisor(q.tiles_y, &q.mul_y, &q.shift_y);
  const std::string key = key_of(d, sh);
  CUfunction fn = nullptr;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (rtc_cached(key, &fn) != PSB_OK) {
    if (gd.interpret) return PSB_ERR_UNSUPPORTED;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
      return PSB_ERR_UNSUPPORTED;  // no compile or module load here
    if (rtc_function(key, source_of(d, sh), "psb_generic_points", {}, 0, &fn) != PSB_OK)
      return PSB_ERR_UNSUPPORTED;
  }
  void *args[] = {&q};
  PSB_CHECK(rtc_launch(fn, (unsigned)(bx * by * bz), kGpThreads, 0, s, args));
  (*launches)++;
  return PSB_OK;
}

}  // namespace psb
