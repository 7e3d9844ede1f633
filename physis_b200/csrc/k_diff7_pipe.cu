// Host side of the multi-step 7-point passes (k_diff7_pipe.cuh).
#include <string.h>

#include <algorithm>
#include <map>

#include "k_diff7_pipe.cuh"

namespace psb {

template <typename T, int NS, int R, int MAXT, int MINB, bool GHOST, bool PERIODIC, bool FAST>
__global__ void __launch_bounds__(MAXT, MINB)
    k_diff7_pipe(const __grid_constant__ CUtensorMap tin, GridView out, int nx, int ny, int nz,
                 C7<T> k, const __grid_constant__ PipeGeom geo, int *err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127);
  diff7_pipe<T, NS, R, GHOST, PERIODIC, FAST>(&tin, out, nx, ny, nz, k, geo, err, smem);
}

// Tiles along one axis: extended tiles of `ext` points, `ns` of them halo on
// each inner side. The first starts at the face (clamped) or `lead` before it
// (periodic: the halo, rounded up to the alignment of a box).
static int pipe_tiles(int n, int ext, int ns, bool periodic, int lead) {
  const int first = periodic ? ext - lead - ns : ext;  // points the first tile finishes alone
  if (first >= n) return 1;
  const int step = ext - 2 * ns;
  return 1 + (n - (periodic ? first : ext) + step - 1) / step;
}

template <typename T, int NS, int R, int MAXT, int MINB, bool PERIODIC, bool FAST>
static psb_status pipe_launch(MapImpl &m, GridImpl *in, GridImpl *out, const PipeConfig &cfg,
                              cudaStream_t s, int64_t *launches) {
  constexpr int V = 16 / (int)sizeof(T);
  const int *n = in->pub.dim;
  PipeGeom g;
  const int xl = 1 << cfg.xl_shift, w = xl * V;
  if (cfg.threads > MAXT || xl > 32 || cfg.threads % 32 || cfg.threads % xl) return PSB_ERR_INVALID;
  g.xl_shift = cfg.xl_shift;
  g.rows = cfg.threads / xl * R;
  g.bx = std::min(w, 256);
  g.nbox = w / g.bx;
  if (g.rows > 256 || g.rows <= 2 * NS || w <= 2 * pipe_hx(NS, V) + V) return PSB_ERR_INVALID;
  const int hx = (NS + V - 1) / V * V;  // periodic tiles start this far before x = 0
  g.ex0 = PERIODIC ? -hx : 0;
  g.ey0 = PERIODIC ? -NS : 0;
  constexpr int HX = pipe_hx(NS, V);
  g.sx = w - 2 * HX;
  g.sy = g.rows - 2 * NS;
  if (g.sx % V) return PSB_ERR_INVALID;
  g.tiles_x = pipe_tiles(n[0], w, HX, PERIODIC, hx);
  g.tiles_y = pipe_tiles(n[1], g.rows, NS, PERIODIC, NS);
  g.zchunk = std::max(1, cfg.zchunk);
  const int nzc = (n[2] + g.zchunk - 1) / g.zchunk;
  g.stages = cfg.stages;
  g.plane_bytes = w * g.rows * (int)sizeof(T);
  g.ax0 = in->pad_left;
  g.ay0 = in->halo;
  g.az0 = in->halo;
  const size_t smem = 128 + 128 + (size_t)g.stages * g.plane_bytes +
                      (size_t)(NS - 1) * 4 * cfg.threads * 16;
  if (g.stages < 3 || g.stages > 16 || smem > rt().smem_optin) return PSB_ERR_INVALID;
  // Faces inside a vector or inside a thread's rows (see GHOST).
  const bool ghost = !PERIODIC && (n[0] % V != 0 || (n[1] < g.rows && n[1] % R != 0));
  auto kern = ghost ? k_diff7_pipe<T, NS, R, MAXT, MINB, !PERIODIC, PERIODIC, FAST>
                    : k_diff7_pipe<T, NS, R, MAXT, MINB, false, PERIODIC, FAST>;
  static bool conf[2] = {false, false};
  bool &configured = conf[ghost];
  if (!configured) {
    PSB_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)rt().smem_optin));
    PSB_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared));
    configured = true;
  }
  const CUtensorMap *map = nullptr;
  PSB_CHECK(get_tmap(in, g.bx, g.rows, &map));
  C7<T> k;
  k.ce = (T)m.params[0];
  k.cw = (T)m.params[1];
  k.cn = (T)m.params[2];
  k.cs = (T)m.params[3];
  k.ct = (T)m.params[4];
  k.cb = (T)m.params[5];
  k.cc = (T)m.params[6];
  const int64_t blocks = (int64_t)g.tiles_x * g.tiles_y * nzc;
  if (blocks > 0x7fffffff) return PSB_ERR_INVALID;
  kern<<<(unsigned)blocks, cfg.threads, smem, s>>>(*map, out->view(), n[0], n[1], n[2], k, g,
                                                   rt().d_error);
  (*launches)++;
  PSB_TRY(cudaGetLastError());
  return PSB_OK;
}

// One pass: cfg.ns steps of map m from grid in to grid out.
psb_status diff7_pipe_launch(MapImpl &m, GridImpl *in, GridImpl *out, const PipeConfig &cfg,
                             cudaStream_t s, int64_t *launches) {
  const bool per = m.kernel_id == PSB_KERNEL_DIFFUSION7_PERIODIC;
  const bool fast = rt().fp_mode == PSB_FP_FMA, dbl = in->pub.elm_size == 8;
#define PSB_PIPE(T, NS, R, MAXT, MINB, PER)                                            \
  (fast ? pipe_launch<T, NS, R, MAXT, MINB, PER, true>(m, in, out, cfg, s, launches)    \
        : pipe_launch<T, NS, R, MAXT, MINB, PER, false>(m, in, out, cfg, s, launches))
  if (cfg.ns == 2 && cfg.r == 4) {
    if (dbl) return per ? PSB_PIPE(double, 2, 4, 192, 2, true) : PSB_PIPE(double, 2, 4, 192, 2, false);
    return per ? PSB_PIPE(float, 2, 4, 192, 2, true) : PSB_PIPE(float, 2, 4, 192, 2, false);
  }
  // More than two steps need more halo than the two cells a periodic grid
  // keeps.
  if (cfg.ns == 4 && cfg.r == 2 && !per)
    return dbl ? PSB_PIPE(double, 4, 2, 384, 1, false) : PSB_PIPE(float, 4, 2, 384, 1, false);
  if (cfg.ns == 3 && cfg.r == 2 && !per)
    return dbl ? PSB_PIPE(double, 3, 2, 384, 1, false) : PSB_PIPE(float, 3, 2, 384, 1, false);
#undef PSB_PIPE
  return PSB_ERR_INVALID;
}

// --------------------------------------------------------------------------
// Choice of the passes' shape. A turn of a walk takes what its SM's warps
// issue (row-stages: one row of one stage of one warp) or the latency of its
// stages, whichever is longer, and `both` of the other; a walk its planes and
// `extra` turns, and in periodic passes the copies of the images after it; a
// pass its full waves of CTAs, the last one and its launch. The constants
// (cycles) are fitted to 10,000 timed shapes (33x40x300 to 512^3 with ragged
// extents): estimates are off by 6 to 12% on average, and the shape chosen
// takes 1 to 4% more than the fastest one timed. Small tiles spread over more
// SMs but recompute more halo.
// --------------------------------------------------------------------------
struct PipeFit {
  double row_stage, latency, both, extra, launch, images;
};

static const PipeFit &pipe_fit(int ns, bool dbl, bool per, bool fast) {
  // [double][FMA]
  static const PipeFit two[2][2] = {{{53.6, 1262, 0.83, 3.1, 8900, 0}, {44.5, 1228, 0.83, 3.1, 7200, 0}},
                                    {{47.5, 916, 0.69, 4.7, 8100, 0}, {43.0, 862, 0.71, 3.9, 7000, 0}}};
  static const PipeFit four[2][2] = {{{32.9, 1280, 0.92, 6.7, 9100, 0}, {31.1, 1015, 0.95, 6.2, 9100, 0}},
                                     {{39.7, 846, 0.81, 9.0, 10800, 0}, {38.5, 783, 0.77, 8.2, 9200, 0}}};
  static const PipeFit wrap[2][2] = {{{75.3, 1595, 0.64, 2.2, 9300, 42}, {49.3, 1693, 0.82, 2.0, 8700, 108}},
                                     {{45.8, 1117, 0.76, 4.1, 9200, 85}, {49.8, 1210, 0.17, 5.5, 7500, 242}}};
  return per ? wrap[dbl][fast] : ns > 2 ? four[dbl][fast] : two[dbl][fast];
}

static double pipe_cost(const PipeConfig &c, bool dbl, bool per, bool fast, const int *n) {
  const int V = dbl ? 2 : 4, w = V << c.xl_shift;
  const int rows = (c.threads >> c.xl_shift) * c.r;
  if (rows <= 2 * c.ns || rows > 256 || w <= 2 * pipe_hx(c.ns, V) + V) return -1;
  const int64_t tiles = (int64_t)pipe_tiles(n[0], w, pipe_hx(c.ns, V), per, (c.ns + V - 1) / V * V) *
                        pipe_tiles(n[1], rows, c.ns, per, c.ns);
  const int64_t blocks = tiles * ((n[2] + c.zchunk - 1) / c.zchunk);
  const size_t smem = 1280 + (size_t)c.stages * w * rows * (dbl ? 8 : 4) +
                      (size_t)(c.ns - 1) * 64 * c.threads;
  const int occ = (int)std::min<size_t>(65536 / (168 * c.threads), (228 << 10) / smem);
  if (occ < 1) return -1;
  const PipeFit &f = pipe_fit(c.ns, dbl, per, fast);
  auto walk = [&](int64_t resident) {  // CTAs on the busiest SM
    const double issue = f.row_stage * c.ns * c.r * std::max(1.0, resident * c.threads / 128.0);
    return (c.zchunk + f.extra) *
               (std::max(issue, f.latency) + f.both * std::min(issue, f.latency)) +
           f.images * c.zchunk * rows / c.threads * resident;
  };
  const int64_t per_wave = (int64_t)rt().sm_count * occ, rest = blocks % per_wave;
  return f.launch + (double)(blocks / per_wave) * walk(occ) +
         (rest ? walk((rest + rt().sm_count - 1) / rt().sm_count) : 0.0);
}

PipeConfig diff7_pipe_choose(int ns, bool dbl, bool per, bool fast, const int *n, double *cost) {
  struct Key {
    int ns, dbl, per, fast, n[3];
    bool operator<(const Key &o) const { return memcmp(this, &o, sizeof(Key)) < 0; }
  };
  static std::map<Key, std::pair<PipeConfig, double>> chosen;  // under the runtime lock
  Key key;
  memset(&key, 0, sizeof(key));
  key.ns = ns;
  key.dbl = dbl;
  key.per = per;
  key.fast = fast;
  for (int i = 0; i < 3; i++) key.n[i] = n[i];
  auto it = chosen.find(key);
  if (it == chosen.end()) {
    PipeConfig best{};
    double best_cost = -1;
    for (int shift = 3; shift <= 5; shift++)
      for (int threads = 64; threads <= (ns > 2 ? 384 : 192); threads += 32) {
        if (threads % (1 << shift)) continue;
        for (int nc = 1; nc <= std::max(1, n[2] / 2) && nc <= 128; nc++) {
          const PipeConfig c{ns, ns > 2 ? 2 : 4, threads, shift, (n[2] + nc - 1) / nc, 4};
          const double t = pipe_cost(c, dbl, per, fast, n);
          if (t > 0 && (best_cost < 0 || t < best_cost)) {
            best = c;
            best_cost = t;
          }
        }
      }
    if (chosen.size() >= 256) chosen.clear();
    it = chosen.emplace(key, std::make_pair(best, best_cost)).first;
  }
  *cost = it->second.second;
  return it->second.first;
}

}  // namespace psb
