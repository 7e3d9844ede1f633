// Batching: many independent grids of uneven sizes advanced together.
//
// A batch member is one double-buffered solve (a 7-point diffusion, clamped
// or periodic, or a Himeno Jacobi relaxation, float) of `steps` steps, i.e.
// what PSStencilRun(m(g0->g1), m(g1->g0), steps/2) does for one grid. The
// work of all members is cut into items -- (member, step, tile) where a tile
// is a 32-, 64- or 128-wide column of the member's domain (the shape that
// fits its extent best) over a z chunk -- and laid out in one device-side
// work list per stencil kind, ordered by step, then member, then tile.
//
// Mode 0 (persistent): one launch per kind with one CTA per resident slot.
// In each CTA a producer thread takes items from the list with an atomic
// cursor, waits for the item's dependencies in the member's previous step
// (the whole step after a residual check or for a small member; otherwise
// the 27 tiles around the item, so a large member's steps overlap like a
// wavefront; acquire loads, bounded waits), passes the item to the consumer
// warps through a small descriptor queue in shared memory and streams its
// input planes by TMA into a ring of stages. The ring is not
// drained between items: the producer runs ahead into the next item's planes
// while the consumers finish the current one, and consumer warps never meet
// at a CTA-wide barrier, so a CTA moves from item to item without a bubble.
// Because the list is ordered by step, every dependency of an item was taken
// before the item itself and the earliest unfinished item can always run:
// the launch needs no co-residency guarantee and cannot deadlock.
// Mode 1 (graph): one launch per step and kind (one item per CTA) over all
// members still running, the sequence captured once in a CUDA graph.
// Mode 2 / 3: the per-grid loop -- each member alone, one launch per step,
// with the plain kernel (the reference's shape) or the tuned TMA kernel.
//
// Items run the same tile arithmetic as the single-grid kernels, so every
// member's result is bit-identical to running it alone. Members may also
// measure a convergence residual every `check_every` steps (7-point:
// |u_{n+1}-u_n|^2 and |u_{n+1}|^2; Himeno: the sum of ss^2) and stop early:
// each consumer warp writes an FP64 partial per item, and the warp that
// completes the last unit of a step combines the partials in index order,
// decides, and only then releases the member's next step, so the decision is
// deterministic and independent of the rest of the batch.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <numeric>
#include <vector>

#include "batch.h"
#include "k_diffusion7.cuh"
#include "k_himeno.cuh"
#include "k_himeno_tb2.cuh"

namespace psb {

// Batched items run 128 consumer threads (4 warps; tile shape per member)
// and one producer warp.
constexpr int kBConsumers = 128;
constexpr int kBWarps = kBConsumers / 32;
constexpr int kBThreads = kBConsumers + 32;
constexpr int kBStages = 6;

// Tile shapes of batched items: t consumer threads along x (4 floats each,
// t = kMinTx .. kMaxTx) by floor(128 / t) thread rows; threads past
// t * floor(128 / t) idle. Each member takes the t that covers its x-y
// extent with the fewest tiles, so narrow grids waste few threads on
// partial tiles (a 50-wide grid uses t = 13, 52 points).
constexpr int kMinTx = 8, kMaxTx = 32;

__host__ __device__ constexpr int stage_bytes_of(int tx_threads, int ty_threads,
                                                 int rows_per_thread) {
  return ((tx_threads * 4 + 8) * (ty_threads * rows_per_thread + 2) * 4 + 127) / 128 * 128;
}

// One ring stride per kernel kind (the largest stage of its shapes): the
// planes of differently shaped tiles follow each other through one ring.
__host__ __device__ constexpr int kind_stage_bytes(int group) {
  int m = 0;
  for (int t = kMinTx; t <= kMaxTx; t++) {
    const int b = stage_bytes_of(t, kBConsumers / t, group == 0 ? kVY : 1);
    m = b > m ? b : m;
  }
  return m;
}

// Himeno items also stream their twelve coefficient tiles by TMA: a second
// ring, one stage per output plane holding field i at i * kCoefTileBytes
// (no tile shape covers more than 512 points).
constexpr int kCoefTileBytes = 512 * 4;
constexpr int kCoefStageBytes = 12 * kCoefTileBytes;
constexpr int kCStages = 3;

// Shared memory of the batched kernel (bytes from the 128-aligned base):
// plane ring barriers full[32] at 0 and empty[32] at 256, item queue
// barriers at 512 (qfull) and 544 (qempty), coefficient ring barriers at 576
// (full) and 640 (empty), item descriptors (kQ x 16 bytes) at 704, plane
// stages from 1280, then (Himeno) the coefficient stages.
constexpr int kQ = 4;  // item descriptors in flight between producer and consumers
constexpr int kSmemRing = 1280;

struct BMember {
  int kind;
  int n[3];
  int tiles_x, tiles_y, nzc, ntiles;
  int steps;        // steps in this launch
  int step0;        // member's global step index at local step 0
  int check_every;  // 0: no checks
  double tol2;      // squared relative tolerance
  const CUtensorMap *tmap[2];
  const CUtensorMap *tcoef;  // Himeno: 12 maps (box TX x TY) of the coefficient fields
  GridView buf[2];
  Dom3 dom;
  C7<float> k7;
  float omega;
  HimenoCoef cf;
  int64_t sy, sz;
  TmaGeom dg;
  HimenoGeom hg;
  double *partials;  // [2][ntiles][kBWarps][2]
  unsigned *step_cnt;   // [steps] warps done in the local step, +1 once it is released
  unsigned *tile_done;  // [ntiles] warps done on the tile, over all steps
  int *stop;         // local steps completed when converged, or -1
  double *res;       // [0] a or gosa, [1] b, [2] gosa of the first check, [3] check count
  int group;         // work list: 0 diffusion, 1 Himeno, 2 Himeno two sweeps per pass
  int cur0;          // buf[cur0] holds the state at local step 0; each unit flips it
  const int *pass_start;  // group 2: local step of each pass (npasses + 1 entries)
  int npasses;
};

struct BatchDev {
  int nmembers;
  const BMember *members;
  const int *order;             // member ids sorted by steps (descending)
  const int64_t *tile_prefix;   // prefix of ntiles over `order`
  const int64_t *step_offset;   // prefix of items over steps
  int max_steps;
  int64_t total_items;
  unsigned long long *cursor;
  int *err;
};

// An item handed from the producer thread to the consumer warps.
struct ItemDesc {
  int m, s, t, flags;
};
enum { kItemEnd = 1, kItemSkip = 2 };
static_assert(704 + kQ * sizeof(ItemDesc) <= kSmemRing, "item descriptors overlap the ring");

__device__ __forceinline__ int upper_index(const int64_t *a, int n, int64_t v) {
  // largest i in [0, n) with a[i] <= v (a non-decreasing, a[0] = 0); the
  // work-list tables are read-only during a launch (non-coherent loads)
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(a + mid) <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ int ld_acquire_int(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Members with at least this many tiles per step wait for the tiles around
// an item of the previous step; smaller ones for the whole previous step.
constexpr int kWaveTiles = 128;

// Warp completions of one step of a member (the last one also releases it).
__device__ __forceinline__ unsigned step_full(const BMember &M) {
  return (unsigned)M.ntiles * kBWarps;
}

// Whether global step gstep measures the residual (and may stop the member).
template <int GROUP>
__device__ __forceinline__ bool is_check_step(const BMember &M, int gstep) {
  return M.check_every > 0 && ((gstep + 1) % M.check_every == 0 || (GROUP == 1 && gstep == 0));
}

__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Output column and planes of item (m, s, t).
struct ItemGeom {
  int x0, y0, zb, nzl;
};

template <int GROUP>
__device__ __forceinline__ ItemGeom item_geom(const BMember &M, int t) {
  const int tiles_x = GROUP == 0 ? M.dg.tiles_x : M.hg.tiles_x;
  const int tiles_y = GROUP == 0 ? M.dg.tiles_y : M.hg.tiles_y;
  const int zchunk = GROUP == 0 ? M.dg.zchunk : M.hg.zchunk;
  const int tx_threads = GROUP == 0 ? M.dg.tx_threads : M.hg.tx_threads;
  const int ty_threads = GROUP == 0 ? M.dg.ty_threads : M.hg.ty_threads;
  const int x_base = GROUP == 0 ? M.dg.x_base : M.hg.x_base;
  const int TX = tx_threads * 4, TY = ty_threads * (GROUP == 0 ? kVY : 1);
  const int tile_x = t % tiles_x;
  const int rest = t / tiles_x;
  const int tile_y = rest % tiles_y;
  const int zc = rest / tiles_y;
  ItemGeom g;
  g.x0 = x_base + tile_x * TX;
  g.y0 = M.dom.lo[1] + tile_y * TY;
  g.zb = M.dom.lo[2] + zc * zchunk;
  g.nzl = min(g.zb + zchunk, M.dom.hi[2]) - g.zb;
  return g;
}

// Dependencies of item (s, t) of member M on its step (or pass) s-1, where
// every item completes `units` counts (one per consumer warp). After a step
// that measures the residual: all of it and its convergence decision.
// Otherwise the tiles this item's planes read (its own and the 26 around
// it, wrapping for periodic members, whose edge tiles also write the
// opposite halo), which are also every tile that read the planes it
// overwrites: consecutive steps of one member overlap like a wavefront
// instead of meeting at a barrier. Every dependency is an item earlier in
// the list, so the earliest unfinished item can always run. Bounded: false
// when the batch's error word is set or the wait gave up.
__device__ bool wait_item_deps(const BatchDev &B, const BMember &M, int s, int t, int units,
                               bool after_check, bool wrap) {
  const unsigned full = (unsigned)M.ntiles * units;
  const unsigned *cnt = M.step_cnt + (s - 1);
  const long long t0 = clock64();
  unsigned sleep = 32;
  if (after_check) {
    while (ld_acquire(cnt) < full + 1u) {
      if (ld_acquire_int(B.err) != 0 || clock64() - t0 > 4000000000LL) return false;
      __nanosleep(sleep);
      if (sleep < 2048) sleep <<= 1;
    }
  } else if (M.ntiles < kWaveTiles) {
    // Small members: their steps are short and end almost together;
    // waiting for the whole step costs one counter.
    while (ld_acquire(cnt) < full) {
      if (ld_acquire_int(B.err) != 0 || clock64() - t0 > 4000000000LL) return false;
      __nanosleep(sleep);
      if (sleep < 2048) sleep <<= 1;
    }
  } else if (ld_acquire(cnt) < full) {
    const int tx = M.tiles_x, ty = M.tiles_y, tz = M.nzc;
    const int cx = t % tx, cy = (t / tx) % ty, cz = t / (tx * ty);
    const unsigned need = (unsigned)s * units;
    // The 27 counters are read together (independent loads in flight at
    // once), then only the ones not yet reached are polled.
    const unsigned *nb[27];
#pragma unroll
    for (int k = 0; k < 27; k++) {
      int x = cx + k % 3 - 1, y = cy + (k / 3) % 3 - 1, z = cz + k / 9 - 1;
      bool in = true;
      if (x < 0 || x >= tx) { in = wrap; x = (x + tx) % tx; }
      if (y < 0 || y >= ty) { in = in && wrap; y = (y + ty) % ty; }
      if (z < 0 || z >= tz) { in = in && wrap; z = (z + tz) % tz; }
      nb[k] = in ? M.tile_done + (x + tx * (y + ty * z)) : nullptr;
    }
    unsigned v[27];
#pragma unroll
    for (int k = 0; k < 27; k++) v[k] = nb[k] ? ld_relaxed(nb[k]) : need;
    unsigned pending = 0;
#pragma unroll
    for (int k = 0; k < 27; k++)
      if (v[k] < need) pending |= 1u << k;
    while (pending) {
      if (ld_acquire_int(B.err) != 0 || clock64() - t0 > 4000000000LL) return false;
      __nanosleep(sleep);
      if (sleep < 2048) sleep <<= 1;
      if (ld_relaxed(cnt) >= full) break;  // the whole step is done
#pragma unroll
      for (int k = 0; k < 27; k++)
        if ((pending >> k & 1u) && ld_relaxed(nb[k]) >= need) pending &= ~(1u << k);
    }
    // Acquire what the relaxed reads observed.
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
  }
  return true;
}

// Producer thread: takes items (from the shared cursor, or item `blockIdx.x`
// of `step` when step >= 0), waits until the item's member has completed
// its previous step, hands the item to the consumers through the descriptor
// queue and streams its input planes into the ring. It runs ahead of the
// consumers by up to the ring's depth, across item boundaries.
template <int GROUP>
__device__ void batch_produce(const BatchDev &B, int step, const Ring &R, const Ring &RC,
                              uint64_t *qfull, uint64_t *qempty, ItemDesc *desc) {
  RingPos pos{0, 0}, cpos{0, 0};
  bool ok = true;
  for (uint32_t nq = 0;; nq++) {
    long long item;
    if (step >= 0)
      item = nq == 0 ? (long long)B.step_offset[step] + blockIdx.x : (long long)B.total_items;
    else
      item = (long long)atomicAdd(B.cursor, 1ull);
    int m = 0, s = 0, t = 0, flags = 0;
    const BMember *M = nullptr;
    if (item >= B.total_items || ld_acquire_int(B.err) != 0) {
      flags = kItemEnd;
    } else {
      s = upper_index(B.step_offset, B.max_steps + 1, item);
      const int64_t local = item - __ldg(B.step_offset + s);
      const int k = upper_index(B.tile_prefix, B.nmembers + 1, local);
      m = __ldg(B.order + k);
      t = (int)(local - __ldg(B.tile_prefix + k));
      M = &B.members[m];
      // Dependencies on step s-1 of the member (wait_item_deps).
      if (s > 0)
        ok = wait_item_deps(B, *M, s, t, kBWarps,
                            is_check_step<GROUP>(*M, M->step0 + s - 1),
                            GROUP == 0 && M->kind == BK_DIFF7P);
      if (!ok) {
        flags = kItemEnd;
      } else {
        const int st = ld_acquire_int(M->stop);
        if (st >= 0 && s >= st) flags = kItemSkip;
      }
    }
    const int q = nq % kQ;
    if (nq >= kQ && !mbar_wait_bounded(&qempty[q], ((nq / kQ) - 1) & 1)) {
      ok = false;
      break;  // the consumers are stuck; their own bounded waits end them
    }
    desc[q].m = m;
    desc[q].s = s;
    desc[q].t = t;
    desc[q].flags = flags;
    mbar_arrive(&qfull[q]);  // release: the descriptor is visible to the consumers
    if (flags & kItemEnd) break;
    if (flags & kItemSkip) continue;
    // The step's inputs were written by generic stores of other CTAs and
    // acquired above; order that before the async-proxy (TMA) reads.
    asm volatile("fence.proxy.async.global;" ::: "memory");
    const int par = (M->cur0 + s) & 1;
    const ItemGeom g = item_geom<GROUP>(*M, t);
    const int bx = GROUP == 0 ? M->dg.bx : M->hg.bx;
    const int by = GROUP == 0 ? M->dg.by : M->hg.by;
    const int ax0 = GROUP == 0 ? M->dg.ax0 : M->hg.ax0;
    const int ay0 = GROUP == 0 ? M->dg.ay0 : M->hg.ay0;
    const int az0 = GROUP == 0 ? M->dg.az0 : M->hg.az0;
    if (GROUP == 0) {
      if (!ring_produce(R, pos, M->tmap[par], (uint32_t)(bx * by * 4), g.x0 - 4 + ax0,
                        g.y0 - 1 + ay0, g.zb - 1 + az0, g.nzl + 2)) {
        ok = false;
        break;
      }
    } else {
      // Himeno: after each plane of p that is also an output plane, the
      // twelve coefficient tiles of that plane into the coefficient ring
      // (the order the consumers need them in, so neither ring can wait on
      // a stage of the other that is not yet issued).
      for (int j = 0; j < g.nzl + 2 && ok; j++) {
        const int z = g.zb - 1 + j;
        ok = ring_produce(R, pos, M->tmap[par], (uint32_t)(bx * by * 4), g.x0 - 4 + ax0,
                          g.y0 - 1 + ay0, z + az0, 1);
        if (ok && z >= g.zb && z < g.zb + g.nzl)
          ok = coef_produce(RC, cpos, M->tcoef, 1, kCoefTileBytes,
                            M->hg.tx_threads * 4 * M->hg.ty_threads * 4, g.x0 + ax0, g.y0 + ay0,
                            z + az0);
      }
      if (!ok) break;
    }
  }
  if (!ok) {
    atomicExch(B.err, 1);
    ring_drain(R, pos);
    if (GROUP == 1) ring_drain(RC, cpos);
  }
}

// Completion of an item by one consumer warp: its FP64 residual partial
// (when the step is checked), then one unit of the tile's and of the step's
// counter. The warp that completes the step's last unit combines the
// partials in index order (deterministic: the same whatever else is in the
// batch), decides convergence, and only then releases the step (the next
// step of a checked one waits for that).
template <int GROUP>
__device__ __forceinline__ void item_done(const BMember &M, int s, int t, int warp, int lane,
                                          bool check, bool contrib, double a, double b) {
  const int par = (M.step0 + s) & 1;
  const int gstep = M.step0 + s;
  double *P = M.partials + (int64_t)par * M.ntiles * kBWarps * 2;
  if (contrib) {
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      P[((int64_t)t * kBWarps + warp) * 2] = a;
      P[((int64_t)t * kBWarps + warp) * 2 + 1] = b;
    }
  }
  __syncwarp();
  unsigned last = 0;
  if (lane == 0) {
    __threadfence();
    atomicAdd(M.tile_done + t, 1u);
    const unsigned old = atomicAdd(M.step_cnt + s, 1u);
    last = old + 1 == step_full(M);
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return;
  if (check && contrib) {
    __threadfence();
    const int n = M.ntiles * kBWarps;
    double sa = 0, sb = 0;
    for (int i = lane; i < n; i += 32) {
      sa += __ldcg(&P[2 * i]);
      sb += __ldcg(&P[2 * i + 1]);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sa += __shfl_down_sync(0xffffffffu, sa, o);
      sb += __shfl_down_sync(0xffffffffu, sb, o);
    }
    if (lane == 0) {
      bool conv;
      if (GROUP == 1) {
        if (gstep == 0) M.res[2] = sa;
        const double g0 = gstep == 0 ? sa : __ldcg(&M.res[2]);
        conv = sa <= M.tol2 * g0;
        M.res[1] = g0;
      } else {
        conv = sa <= M.tol2 * sb;
        M.res[1] = sb;
      }
      M.res[0] = sa;
      M.res[3] = (double)(gstep + 1);
      if (conv && M.tol2 > 0) atomicExch(M.stop, s + 1);
    }
  }
  if (lane == 0) {
    __threadfence();
    atomicAdd(M.step_cnt + s, 1u);
  }
}

// Consumer warps: take item after item from the descriptor queue and run
// the tile's computation from the rings.
template <int GROUP>
__device__ void batch_consume(const BatchDev &B, const Ring &R, const Ring &RC, uint64_t *qfull,
                              uint64_t *qempty, const ItemDesc *desc) {
  RingPos pos{0, 0}, cpos{0, 0};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t nq = 0;; nq++) {
    const int q = nq % kQ;
    const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&qfull[q], (nq / kQ) & 1));
    if (!got) {
      if (lane == 0) atomicExch(B.err, 1);
      return;
    }
    const int dm = desc[q].m, ds = desc[q].s, dt = desc[q].t, dflags = desc[q].flags;
    if (dflags & kItemEnd) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&qempty[q]);
      return;
    }
    const BMember &M = B.members[dm];
    const bool skip = (dflags & kItemSkip) != 0;
    const int par = (M.cur0 + ds) & 1;
    __syncwarp();
    if (lane == 0) mbar_arrive(&qempty[q]);
    const bool check = is_check_step<GROUP>(M, M.step0 + ds);
    double a = 0, b = 0;
    if (!skip) {
      const ItemGeom g = item_geom<GROUP>(M, dt);
      bool ok;
      if constexpr (GROUP == 1) {
        ok = himeno_consume_staged(R, pos, RC, cpos, kCoefTileBytes, (float *)M.buf[par ^ 1].origin,
                                   M.sy, M.sz, M.dom, M.omega, M.hg, g.x0, g.y0, g.zb, g.nzl, &a);
      } else {
        TileAcc acc{0, 0};
        const GridView out = M.buf[par ^ 1];
        if (M.kind == BK_DIFF7P) {
          ok = check ? diff7_consume<float, true, true>(R, pos, out, M.n[0], M.n[1], M.n[2], M.dom,
                                                        M.k7, M.dg, g.x0, g.y0, g.zb, g.nzl, 1,
                                                        &acc)
                     : diff7_consume<float, true, false>(R, pos, out, M.n[0], M.n[1], M.n[2],
                                                         M.dom, M.k7, M.dg, g.x0, g.y0, g.zb,
                                                         g.nzl, 1, nullptr);
        } else {
          ok = check ? diff7_consume<float, false, true>(R, pos, out, M.n[0], M.n[1], M.n[2],
                                                         M.dom, M.k7, M.dg, g.x0, g.y0, g.zb,
                                                         g.nzl, 0, &acc)
                     : diff7_consume<float, false, false>(R, pos, out, M.n[0], M.n[1], M.n[2],
                                                          M.dom, M.k7, M.dg, g.x0, g.y0, g.zb,
                                                          g.nzl, 0, nullptr);
        }
        a = acc.a;
        b = acc.b;
      }
      if (!ok) {
        if (lane == 0) atomicExch(B.err, 1);
        return;
      }
    }
    item_done<GROUP>(M, ds, dt, warp, lane, check, check && !skip, a, b);
  }
}

__device__ __forceinline__ unsigned char *aligned_smem(unsigned char *raw) {
  return raw + ((128 - (smem_u32(raw) & 127)) & 127);
}

// The batched kernel of one stencil kind. step < 0: persistent -- each CTA
// takes items from the kind's work list until it is exhausted (mode 0).
// step >= 0: one item per CTA, item blockIdx.x of that step (mode 1, one
// launch per step). Diffusion items run 3 CTAs per SM; Himeno items, whose
// CTAs also hold three stages of coefficient tiles (72 KB), run 2.
template <int GROUP>
__global__ void __launch_bounds__(kBThreads, GROUP == 0 ? 3 : 2) k_batch(BatchDev B, int step) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = aligned_smem(smem_raw);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  uint64_t *qfull = bars + 64, *qempty = bars + 68;
  ItemDesc *desc = reinterpret_cast<ItemDesc *>(smem + 704);
  const Ring R{bars, bars + 32, smem + kSmemRing, kBStages, kind_stage_bytes(GROUP)};
  const Ring RC{bars + 72, bars + 80, smem + kSmemRing + kBStages * kind_stage_bytes(GROUP),
                kCStages, kCoefStageBytes};
  if (threadIdx.x == 0) {
    ring_init(R, kBWarps);
    if (GROUP == 1) ring_init(RC, kBWarps);
    for (int q = 0; q < kQ; q++) {
      mbar_init(&qfull[q], 1);
      mbar_init(&qempty[q], kBWarps);
    }
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x >= kBConsumers) {
    if (threadIdx.x == kBConsumers) batch_produce<GROUP>(B, step, R, RC, qfull, qempty, desc);
    return;
  }
  batch_consume<GROUP>(B, R, RC, qfull, qempty, desc);
}

// ---------------------------------------------------------------------------
// Group 2: Himeno members that advance up to two sweeps per item (passes).
//
// A member's local steps are cut into passes of one or two sweeps
// (pass_start); a pass never straddles a residual check (a check step is
// always the last step of its pass), so a check sees the sweep it needs.
// Items are (member, pass, 64 x 12 tile x z chunk); the work list is ordered
// by pass, then member, then tile, and an item depends on pass - 1 of its
// member exactly as a single-sweep item depends on step - 1 (wait_item_deps:
// the two-sweep halo of 2 cells stays inside the 27 tiles around it). Each
// pass flips which buffer holds the state (buf[(cur0 + pass) & 1] in,
// buf[(cur0 + pass + 1) & 1] out), so a two-sweep pass never writes the
// buffer it reads. A CTA is one producer thread, seven first-sweep warps, six
// second-sweep warps and the edge warp on the rings of k_himeno_tb2.cuh; a one-sweep
// pass runs the same rings with the second stage storing the first sweep.
// Every consumer warp completes one unit per item (thirteen per item;
// the edge warp none).
// ---------------------------------------------------------------------------
constexpr int kT2Units = kHtW1 + kHtW2;
constexpr int kT2Threads = 32 * (1 + kT2Units + 1);  // and the edge warp
constexpr int kT2SmemRing = 1024;
constexpr size_t kT2Smem = 128 + kT2SmemRing + kHtRingBytes;

__device__ __forceinline__ int pass_end(const BMember &M, int q) { return __ldg(M.pass_start + q + 1); }

// Whether pass q of a group-2 member ends with a residual check.
__device__ __forceinline__ bool pass_checked(const BMember &M, int q) {
  return is_check_step<1>(M, M.step0 + pass_end(M, q) - 1);
}

// Geometry of item t of a group-2 member: 64 x 12 tiles over the interior.
__device__ __forceinline__ void t2_geom(const BMember &M, int t, int &x0, int &y0, int &zb,
                                        int &nzl) {
  const int tile_x = t % M.tiles_x;
  const int rest = t / M.tiles_x;
  const int tile_y = rest % M.tiles_y;
  const int zc = rest / M.tiles_y;
  x0 = M.hg.x_base + tile_x * kHtTX;
  y0 = M.dom.lo[1] + tile_y * kHtTY;
  zb = M.dom.lo[2] + zc * M.hg.zchunk;
  nzl = min(zb + M.hg.zchunk, M.dom.hi[2]) - zb;
}

__device__ void t2_produce(const BatchDev &B, int step, const HtRings &R, uint64_t *qfull,
                           uint64_t *qempty, ItemDesc *desc) {
  RingPos p1{0, 0}, pc{0, 0};
  bool ok = true;
  for (uint32_t nq = 0;; nq++) {
    long long item;
    if (step >= 0)
      item = nq == 0 ? (long long)B.step_offset[step] + blockIdx.x : (long long)B.total_items;
    else
      item = (long long)atomicAdd(B.cursor, 1ull);
    int m = 0, s = 0, t = 0, flags = 0;
    const BMember *M = nullptr;
    if (item >= B.total_items || ld_acquire_int(B.err) != 0) {
      flags = kItemEnd;
    } else {
      s = upper_index(B.step_offset, B.max_steps + 1, item);
      const int64_t local = item - __ldg(B.step_offset + s);
      const int k = upper_index(B.tile_prefix, B.nmembers + 1, local);
      m = __ldg(B.order + k);
      t = (int)(local - __ldg(B.tile_prefix + k));
      M = &B.members[m];
      if (s > 0) ok = wait_item_deps(B, *M, s, t, kT2Units, pass_checked(*M, s - 1), false);
      if (!ok) {
        flags = kItemEnd;
      } else {
        const int st = ld_acquire_int(M->stop);
        if (st >= 0 && __ldg(M->pass_start + s) >= st) flags = kItemSkip;
      }
    }
    const int q = nq % kQ;
    if (nq >= kQ && !mbar_wait_bounded(&qempty[q], ((nq / kQ) - 1) & 1)) {
      ok = false;
      break;
    }
    desc[q].m = m;
    desc[q].s = s;
    desc[q].t = t;
    desc[q].flags = flags;
    mbar_arrive(&qfull[q]);
    if (flags & kItemEnd) break;
    if (flags & kItemSkip) continue;
    asm volatile("fence.proxy.async.global;" ::: "memory");
    const int par = (M->cur0 + s) & 1;
    int x0, y0, zb, nzl;
    t2_geom(*M, t, x0, y0, zb, nzl);
    if (!ht_produce_tile(R, p1, pc, M->tmap[par], M->tcoef, M->hg.ax0, M->hg.ay0, M->hg.az0, x0,
                         y0, zb, nzl)) {
      ok = false;
      break;
    }
  }
  if (!ok) {
    atomicExch(B.err, 1);
    ht_drain(R, p1, pc);
  }
}

// Completion of a group-2 item by consumer warp cw (0..12): its FP64
// residual partial when the pass ends with a check, one unit of the tile's
// and of the pass's counter; the warp that completes the pass combines the
// partials in index order, decides, and only then releases the pass.
__device__ __forceinline__ void t2_item_done(const BMember &M, int q, int t, int cw, int lane,
                                             bool check, bool contrib, double a) {
  const int pend = pass_end(M, q);
  const int gstep = M.step0 + pend - 1;
  double *P = M.partials + (int64_t)(q & 1) * M.ntiles * kT2Units * 2;
  if (contrib) {
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) {
      P[((int64_t)t * kT2Units + cw) * 2] = a;
      P[((int64_t)t * kT2Units + cw) * 2 + 1] = 0.0;
    }
  }
  __syncwarp();
  unsigned last = 0;
  if (lane == 0) {
    __threadfence();
    atomicAdd(M.tile_done + t, 1u);
    const unsigned old = atomicAdd(M.step_cnt + q, 1u);
    last = old + 1 == (unsigned)M.ntiles * kT2Units;
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return;
  if (check && contrib) {
    __threadfence();
    const int n = M.ntiles * kT2Units;
    double sa = 0;
    for (int i = lane; i < n; i += 32) sa += __ldcg(&P[2 * i]);
    for (int o = 16; o > 0; o >>= 1) sa += __shfl_down_sync(0xffffffffu, sa, o);
    if (lane == 0) {
      if (gstep == 0) M.res[2] = sa;
      const double g0 = gstep == 0 ? sa : __ldcg(&M.res[2]);
      const bool conv = sa <= M.tol2 * g0;
      M.res[1] = g0;
      M.res[0] = sa;
      M.res[3] = (double)(gstep + 1);
      if (conv && M.tol2 > 0) atomicExch(M.stop, pend);
    }
  }
  if (lane == 0) {
    __threadfence();
    atomicAdd(M.step_cnt + q, 1u);
  }
}

__device__ void t2_consume(const BatchDev &B, const HtRings &R, uint64_t *qfull,
                           uint64_t *qempty, const ItemDesc *desc) {
  const int lane = threadIdx.x & 31, cw = (threadIdx.x >> 5) - 1;
  const bool first = cw < kHtW1;
  RingPos p1{0, 0}, pc{0, 0}, p2{0, 0};
  for (uint32_t nq = 0;; nq++) {
    const int q = nq % kQ;
    const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&qfull[q], (nq / kQ) & 1));
    if (!got) {
      if (lane == 0) atomicExch(B.err, 1);
      return;
    }
    const int dm = desc[q].m, ds = desc[q].s, dt = desc[q].t, dflags = desc[q].flags;
    __syncwarp();
    if (lane == 0) mbar_arrive(&qempty[q]);
    if (dflags & kItemEnd) return;
    const BMember &M = B.members[dm];
    const bool skip = (dflags & kItemSkip) != 0;
    const int len = pass_end(M, ds) - __ldg(M.pass_start + ds);
    const bool check = pass_checked(M, ds);
    double a = 0.0;
    if (!skip) {
      int x0, y0, zb, nzl;
      t2_geom(M, dt, x0, y0, zb, nzl);
      bool ok;
      if (cw == kT2Units) {
        ok = ht_edge_tile<false>(R, p1, pc, p2, lane, M.dom, M.omega, x0, y0, zb, nzl);
      } else if (first) {
        ok = ht_stage1_tile<false>(R, p1, pc, p2, threadIdx.x - 32, lane, M.dom, M.omega, x0, y0,
                                   zb, nzl, check && len == 1, &a);
      } else {
        const int par = (M.cur0 + ds) & 1;
        ok = ht_stage2_tile(R, p2, pc, threadIdx.x - 32 - 32 * kHtW1, lane,
                            (float *)M.buf[par ^ 1].origin, M.sy, M.sz, M.dom, M.omega, x0, y0,
                            zb, nzl, len == 1, check && len == 2, &a);
      }
      if (!ok) {
        if (lane == 0) atomicExch(B.err, 1);
        return;
      }
    }
    // The edge warp's points reach the output through the second-sweep warps,
    // which complete the item.
    if (cw < kT2Units) t2_item_done(M, ds, dt, cw, lane, check, check && !skip, a);
  }
}

// The group-2 kernel. step < 0: persistent (mode 0); step >= 0: item
// blockIdx.x of that pass (mode 1). One CTA per SM (its rings take 223 KB).
__global__ void __launch_bounds__(kT2Threads, 1) k_batch_tb2(BatchDev B, int step) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = aligned_smem(smem_raw);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  const HtRings R = ht_rings(bars, smem + kT2SmemRing);
  uint64_t *qfull = bars + 48, *qempty = bars + 52;
  ItemDesc *desc = reinterpret_cast<ItemDesc *>(smem + 448);
  if (threadIdx.x == 0) {
    ht_init(R);
    for (int q = 0; q < kQ; q++) {
      mbar_init(&qfull[q], 1);
      mbar_init(&qempty[q], kT2Units + 1);
    }
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) t2_produce(B, step, R, qfull, qempty, desc);
    return;
  }
  t2_consume(B, R, qfull, qempty, desc);
}
static_assert(448 + kQ * sizeof(ItemDesc) <= kT2SmemRing, "item descriptors overlap the rings");

}  // namespace psb

using namespace psb;

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Work list of one kernel kind (group 0: diffusion members, 1: Himeno).
struct BatchGroup {
  std::vector<int> order;               // member ids of this group, by steps (descending)
  std::vector<int64_t> tile_prefix, step_offset;
  int max_steps = 0;
  int64_t total_items = 0;
  int *d_order = nullptr;
  int64_t *d_tile_prefix = nullptr;
  int64_t *d_step_offset = nullptr;
  unsigned long long *d_cursor = nullptr;
  size_t cap_order = 0, cap_tile_prefix = 0, cap_step_offset = 0;
  int blocks_persistent = 0;
  double work = 0;  // algorithmic bytes of the list (orders the concurrent launches)
};

struct psb_batch {
  std::vector<BatchMemberHost> hm;
  std::vector<double> res_init;  // 4 per member, uploaded by batch_prepare when set
  BMember *d_members = nullptr;
  CUtensorMap *d_tmaps = nullptr;
  double *d_partials = nullptr;
  unsigned *d_done = nullptr;  // per member: step counters, then tile counters
  int64_t n_counters = 1;
  int *d_stop = nullptr;
  double *d_res = nullptr;
  size_t cap_members = 0, cap_tmaps = 0, cap_partials = 0, cap_done = 0, cap_stop = 0,
         cap_res = 0;  // bytes allocated (device buffers are reused while they fit)
  std::vector<BMember> members;
  BatchGroup grp[3];
  std::vector<std::vector<int>> passes;  // group-2 members: local step of each pass
  int *d_pass = nullptr;
  size_t cap_pass = 0;
  int *d_rims = nullptr;  // batch_check_rims: one word per member that it looks at
  size_t cap_rims = 0;
  bool built = false;
  cudaGraphExec_t graph = nullptr;
  cudaStream_t side = nullptr, side2 = nullptr;  // streams of the second and third work lists
  cudaEvent_t fork = nullptr, join = nullptr, join2 = nullptr;
  double last_ms = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;  // batch timing (apart from PSStencilRun's)
  int64_t last_launches = 0;
  int64_t last_lups = 0;
};

namespace psb {



// The work lists and descriptors no longer match the members.
static void batch_invalidate(psb_batch *b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  b->graph = nullptr;
  b->built = false;
}

static void batch_release_device(psb_batch *b) {
  batch_invalidate(b);
  cudaFree(b->d_members);
  cudaFree(b->d_tmaps);
  cudaFree(b->d_partials);
  cudaFree(b->d_done);
  cudaFree(b->d_stop);
  cudaFree(b->d_res);
  cudaFree(b->d_pass);
  b->d_pass = nullptr;
  b->cap_pass = 0;
  cudaFree(b->d_rims);
  b->d_rims = nullptr;
  b->cap_rims = 0;
  b->d_members = nullptr;
  b->d_tmaps = nullptr;
  b->d_partials = nullptr;
  b->d_done = nullptr;
  b->d_stop = nullptr;
  b->d_res = nullptr;
  b->cap_members = b->cap_tmaps = b->cap_partials = b->cap_done = b->cap_stop = b->cap_res = 0;
  for (auto &g : b->grp) {
    cudaFree(g.d_order);
    cudaFree(g.d_tile_prefix);
    cudaFree(g.d_step_offset);
    cudaFree(g.d_cursor);
    g = BatchGroup();
  }
}

// Make *p hold at least `bytes` (grown by half again when it must grow, so
// a server's changing member list rarely reallocates).
template <typename T>
static psb_status dev_reserve(T **p, size_t *cap, size_t bytes) {
  bytes = std::max<size_t>(bytes, 16);
  if (bytes <= *cap) return PSB_OK;
  const size_t want = std::max(bytes, *cap + *cap / 2);
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  PSB_TRY(device_malloc(p, want));
  *cap = want;
  return PSB_OK;
}

// Each member takes the tile shape with the fewest tiles over its x-y
// extent (then the fewest box elements), so small and narrow members waste
// few threads on partial tiles.
#ifndef PSB_PROMO_P
#define PSB_PROMO_P CU_TENSOR_MAP_L2_PROMOTION_L2_256B
#endif
#ifndef PSB_PROMO_C
#define PSB_PROMO_C CU_TENSOR_MAP_L2_PROMOTION_L2_128B
#endif
#ifndef PSB_PROMO_D
#define PSB_PROMO_D CU_TENSOR_MAP_L2_PROMOTION_L2_256B
#endif
// L2 promotion of the batched kernels' tensor maps. Coefficient tiles start
// 128 bytes into a 256-byte line, so promoting their rows to 256 bytes
// fetches lines that small members never use (measured: 128-byte
// promotion is up to 14% faster on small Himeno members).
static const int kPromoP = PSB_PROMO_P, kPromoC = PSB_PROMO_C, kPromoD = PSB_PROMO_D;

// Tile width and z-chunk preference of a member: forced by an autotuner
// trial, else the tuned entry of its size bucket, else none (0: the rules
// below decide).
struct MemberTune {
  int tx = 0;
  int zc = 0;
  int td = 1;  // Himeno sweeps per pass
  bool forced = false;
  bool tuned = false;  // from the bucket's tune entry (tx 0: the entry kept the rule)
};

static MemberTune member_tune(const BatchMemberHost &h) {
  MemberTune t;
  if (h.force_tx > 0 || h.force_zc > 0 || h.force_td > 0) {
    t.tx = h.force_tx;
    t.zc = h.force_zc;
    t.td = h.force_td > 0 ? h.force_td : 1;
    t.forced = true;
    return t;
  }
  psb_tune_config c;
  if (batch_tune_find(h.kind, h.grids[0]->pub.dim, &c)) {
    t.tuned = true;
    t.tx = c.tile_x / 4;
    t.zc = c.z_chunk;
    t.td = c.t_depth;
  }
  return t;
}

// Sweeps per pass of a Himeno member whose bucket has no tune entry: two
// when it is at least 120 points inside on every axis and the 64-wide tiles
// of the two-sweep pass leave at most 15% of their columns outside its x
// extent. Persistent batch, ms per 20 steps, one sweep / two: cubes of 256
// 2.92 / 2.29, 240 2.58 / 1.95, 224 1.99 / 1.72, 192 1.35 / 1.14, 176 1.20 /
// 0.97, 128 0.54 / 0.50; cubes of 160 and 144, which waste 18 and 26% of the
// columns, 0.81 / 1.08 and 0.78 / 0.85; (70, 70, 140) 0.24 / 0.30. Several
// members on the two-sweep list gain more (eight cubes of 128 2.99 / 2.43).
// One beside small members on the other lists gains from 240 on (3.12 / 2.79
// at 256), loses 2 to 13% between 176 and 224 and 27% at 128: the two lists'
// blocks share the SMs badly. The shipped table keeps one sweep in every bucket
// of at most 128 in some extent; the bucket of 129 to 256 has no entry, because
// both answers occur in it.
static int default_sweeps(const BatchMemberHost &h) {
  const int *n = h.grids[0]->pub.dim;
  const int ix = n[0] - 2, iy = n[1] - 2, iz = n[2] - 2;
  if (ix < 120 || iy < 120 || iz < 120) return 1;
  const int cols = (n[0] - 1 + kHtTX - 1) / kHtTX * kHtTX;  // columns of batch_t2geom's tiles
  return ix * 100 >= cols * 85 ? 2 : 1;
}

// Work list of a member: 0 diffusion, 1 Himeno one sweep per item, 2 Himeno
// up to two sweeps per item (when its tune entry or trial says so, or, with
// neither, default_sweeps; and it runs at least two steps, with no coefficient
// that is one of its pressure grids: a pass reads coefficients once for both
// sweeps. Nor where those two hold different values around the domain: a pass
// takes its input's for both sweeps and leaves out every other grid).
static bool two_sweep_member(const BatchMemberHost &h, const MemberTune &mt, int steps) {
  if (h.kind != BK_HIMENO || steps < 2) return false;
  for (int i = 2; i < 14; i++)
    if (h.grids[i] == h.grids[0] || h.grids[i] == h.grids[1]) return false;
  return (mt.tuned || mt.forced ? mt.td : default_sweeps(h)) == 2;
}

static int member_group(const BatchMemberHost &h, const MemberTune &mt, int steps) {
  if (h.kind != BK_HIMENO) return 0;
  return two_sweep_member(h, mt, steps) && !h.rims_differ ? 2 : 1;
}

// Passes of a group-2 member: from each local step s (global step0 + s) two
// sweeps unless s is a check step or the last step, so that every check
// step ends its pass.
static std::vector<int> member_passes(const BatchMemberHost &h, int step0, int steps) {
  std::vector<int> st{0};
  auto check = [&](int g) {
    return h.check_every > 0 && ((g + 1) % h.check_every == 0 || g == 0);
  };
  int s = 0;
  while (s < steps) {
    s += (s + 1 < steps && !check(step0 + s)) ? 2 : 1;
    st.push_back(s);
  }
  return st;
}

static void pick_shape(int nx, int ny, int rows_per_thread, int *tx_threads, int *ty_threads,
                       int force_t = 0) {
  if (force_t >= kMinTx && force_t <= kMaxTx) {
    *tx_threads = force_t;
    *ty_threads = kBConsumers / force_t;
    return;
  }
  int64_t best_tiles = -1, best_box = 0;
  for (int t = kMinTx; t <= kMaxTx; t++) {
    const int TX = t * 4, TY = (kBConsumers / t) * rows_per_thread;
    const int64_t tiles = (int64_t)((nx + TX - 1) / TX) * ((ny + TY - 1) / TY);
    const int64_t box = tiles * (TX + 8) * (TY + 2);
    if (best_tiles < 0 || tiles < best_tiles || (tiles == best_tiles && box < best_box)) {
      best_tiles = tiles;
      best_box = box;
      *tx_threads = t;
      *ty_threads = kBConsumers / t;
    }
  }
}

// Planes per item. The members of a kind together should give enough items
// per step for several waves of CTAs (items_target()); each item's fixed
// costs (a descriptor, a dependency check, two halo planes) favour long
// chunks. So the kind takes the longest chunk `floor` (64 down to 4) at
// which its members together reach the target, and a member whose own
// steps reach it with a longer chunk takes that one: a few large members
// are not quantised into a fraction of a wave at every step, many small
// members are not cut finer than the batch needs, and a lone small
// member's steps (a chain of dependent launches' worth of work) stay short.
static int64_t items_target() { return (int64_t)rt().sm_count * 6; }

static int pick_zchunk(int64_t tiles_xy, int nz, int floor) {
  for (int zc = 64; zc > floor; zc >>= 1)
    if (tiles_xy * ((nz + zc - 1) / zc) >= items_target()) return zc;
  return floor;
}

// z chunk of a member: the trial's, else the longest chunk from the batch's
// floor that reaches the items target. A tuned entry's chunk is not used
// here: the chunk that keeps every SM busy depends on what else is in the
// batch, which the floor accounts for (measured: raising the floor to the
// tuned chunks made the 256-member batch 11% slower).
static int member_zchunk(const MemberTune &mt, int64_t tiles_xy, int nz, int zc_floor) {
  if (mt.forced && mt.zc > 0) return mt.zc;
  return pick_zchunk(tiles_xy, nz, zc_floor);
}

static TmaGeom batch_dgeom(const GridImpl *g, int zc_floor, const MemberTune &mt) {
  TmaGeom geo;
  pick_shape(g->pub.dim[0], g->pub.dim[1], kVY, &geo.tx_threads, &geo.ty_threads, mt.tx);
  const int TX = geo.tx_threads * 4, TY = geo.ty_threads * kVY;
  geo.bx = TX + 8;
  geo.by = TY + 2;
  geo.ax0 = g->pad_left;
  geo.ay0 = g->halo;
  geo.az0 = g->halo;
  geo.x_base = 0;
  geo.tiles_x = (g->pub.dim[0] + TX - 1) / TX;
  geo.tiles_y = (g->pub.dim[1] + TY - 1) / TY;
  geo.zchunk = member_zchunk(mt, (int64_t)geo.tiles_x * geo.tiles_y, g->pub.dim[2], zc_floor);
  geo.stages = kBStages;
  geo.stage_bytes = kind_stage_bytes(0);
  return geo;
}

static HimenoGeom batch_hgeom(const GridImpl *g, int zc_floor, const MemberTune &mt) {
  HimenoGeom geo;
  // interior domain [1, n-1): tiles start at x = 0 (x_base), y = 1.
  pick_shape(g->pub.dim[0] - 1, g->pub.dim[1] - 2, 1, &geo.tx_threads, &geo.ty_threads, mt.tx);
  const int TX = geo.tx_threads * 4, TY = geo.ty_threads;
  geo.bx = TX + 8;
  geo.by = TY + 2;
  geo.ax0 = g->pad_left;
  geo.ay0 = g->halo;
  geo.az0 = g->halo;
  geo.x_base = 0;
  geo.tiles_x = (g->pub.dim[0] - 1 + TX - 1) / TX;
  geo.tiles_y = (g->pub.dim[1] - 2 + TY - 1) / TY;
  geo.zchunk = member_zchunk(mt, (int64_t)geo.tiles_x * geo.tiles_y, g->pub.dim[2] - 2, zc_floor);
  geo.stages = kBStages;
  geo.stage_bytes = kind_stage_bytes(1);
  geo.nx = g->pub.dim[0];
  return geo;
}

// Group 2: 64 x 12 tiles over the interior [1, n-1), x from 0; the pressure
// box (72 x 16) is the tensor-map box of the member's p grids.
static HimenoGeom batch_t2geom(const GridImpl *g, int zc_floor, const MemberTune &mt) {
  HimenoGeom geo;
  geo.tx_threads = kHtTX / 4;
  geo.ty_threads = kHtTY;
  geo.bx = kHtBX;
  geo.by = kHtBY1;
  geo.ax0 = g->pad_left;
  geo.ay0 = g->halo;
  geo.az0 = g->halo;
  geo.x_base = 0;
  geo.tiles_x = (g->pub.dim[0] - 1 + kHtTX - 1) / kHtTX;
  geo.tiles_y = (g->pub.dim[1] - 2 + kHtTY - 1) / kHtTY;
  geo.zchunk = member_zchunk(mt, (int64_t)geo.tiles_x * geo.tiles_y, g->pub.dim[2] - 2, zc_floor);
  geo.stages = kHtS1;
  geo.stage_bytes = kHtStage1;
  geo.nx = g->pub.dim[0];
  return geo;
}

static size_t batch_smem(int group) {
  if (group == 2) return kT2Smem;
  return 128 + kSmemRing + (size_t)kBStages * kind_stage_bytes(group) +
         (group == 1 ? (size_t)kCStages * kCoefStageBytes : 0);
}

// Build the device work lists and member descriptors for one launch in which
// member i runs steps[i] steps starting at its global step step0[i].
psb_status batch_prepare(psb_batch *b, const std::vector<int> &steps, const std::vector<int> &step0) {
  Runtime &r = rt();
  const int n = (int)b->hm.size();
  batch_invalidate(b);
  b->members.assign(n, BMember());
  std::vector<CUtensorMap> tmaps(2 * std::max(1, n));
  std::vector<int> coef_map(n, -1);  // index of a Himeno member's 12 coefficient maps
  std::vector<MemberTune> mt(n);
  std::vector<int> group(n), units(n);  // work list and its units (steps or passes) per member
  b->passes.assign(n, std::vector<int>());
  for (int i = 0; i < n; i++) {
    mt[i] = member_tune(b->hm[i]);
    group[i] = member_group(b->hm[i], mt[i], steps[i]);
    units[i] = std::max(0, steps[i]);
    if (group[i] == 2) {
      b->passes[i] = member_passes(b->hm[i], step0[i], steps[i]);
      units[i] = (int)b->passes[i].size() - 1;
    }
  }
  // The longest z chunk at which each work list's members together give
  // items_target() items per step (4 if none does).
  auto xy_tiles = [&](int i, int k) -> int64_t {
    const GridImpl *g0 = b->hm[i].grids[0];
    if (k == 2) {
      const HimenoGeom hg = batch_t2geom(g0, 64, mt[i]);
      return (int64_t)hg.tiles_x * hg.tiles_y;
    }
    if (k == 1) {
      const HimenoGeom hg = batch_hgeom(g0, 64, mt[i]);
      return (int64_t)hg.tiles_x * hg.tiles_y;
    }
    const TmaGeom dg = batch_dgeom(g0, 64, mt[i]);
    return (int64_t)dg.tiles_x * dg.tiles_y;
  };
  int zc_floor[3] = {4, 4, 4};
  for (int k = 0; k < 3; k++) {
    for (int zc = 64; zc > 4; zc >>= 1) {
      int64_t items = 0;
      for (int i = 0; i < n; i++) {
        if (steps[i] <= 0 || group[i] != k) continue;
        const int nz = b->hm[i].grids[0]->pub.dim[2] - (k == 0 ? 0 : 2);
        items += xy_tiles(i, k) * ((nz + zc - 1) / zc);
      }
      if (items >= items_target()) {
        zc_floor[k] = zc;
        break;
      }
    }
  }
  int64_t partial_slots = 0, pass_words = 0;
  for (int i = 0; i < n; i++) {
    const BatchMemberHost &h = b->hm[i];
    BMember &M = b->members[i];
    memset(&M, 0, sizeof(M));
    M.kind = h.kind;
    M.group = group[i];
    GridImpl *g0 = h.grids[0], *g1 = h.grids[1];
    for (int k = 0; k < 3; k++) M.n[k] = g0->pub.dim[k];
    M.steps = steps[i];
    M.step0 = step0[i];
    M.cur0 = h.cur0 & 1;
    M.check_every = h.check_every;
    M.tol2 = h.tol * h.tol;
    M.buf[0] = g0->view();
    M.buf[1] = g1->view();
    M.sy = g0->sy;
    M.sz = g0->sz;
    const CUtensorMap *a = nullptr, *c = nullptr;
    if (h.kind == BK_HIMENO) {
      const bool two = group[i] == 2;
      M.hg = two ? batch_t2geom(g0, zc_floor[2], mt[i]) : batch_hgeom(g0, zc_floor[1], mt[i]);
      for (int k = 0; k < 3; k++) {
        M.dom.lo[k] = 1;
        M.dom.hi[k] = g0->pub.dim[k] - 1;
      }
      M.tiles_x = M.hg.tiles_x;
      M.tiles_y = M.hg.tiles_y;
      M.nzc = (g0->pub.dim[2] - 2 + M.hg.zchunk - 1) / M.hg.zchunk;
      M.omega = (float)h.params[0];
      for (int k = 0; k < 12; k++) M.cf.f[k] = (const float *)h.grids[2 + k]->view().origin;
      PSB_CHECK(get_tmap(g0, M.hg.bx, M.hg.by, &a, kPromoP));
      PSB_CHECK(get_tmap(g1, M.hg.bx, M.hg.by, &c, kPromoP));
      coef_map[i] = (int)tmaps.size();
      for (int k = 0; k < 12; k++) {
        const CUtensorMap *cm = nullptr;
        if (two)
          PSB_CHECK(get_tmap(h.grids[2 + k], kHtBX, kHtBY2, &cm, kPromoC));
        else
          PSB_CHECK(get_tmap(h.grids[2 + k], M.hg.tx_threads * 4, M.hg.ty_threads, &cm, kPromoC));
        tmaps.push_back(*cm);
      }
      if (two) {
        M.npasses = units[i];
        pass_words += units[i] + 1;
      }
    } else {
      M.dg = batch_dgeom(g0, zc_floor[0], mt[i]);
      for (int k = 0; k < 3; k++) {
        M.dom.lo[k] = 0;
        M.dom.hi[k] = g0->pub.dim[k];
      }
      M.tiles_x = M.dg.tiles_x;
      M.tiles_y = M.dg.tiles_y;
      M.nzc = (g0->pub.dim[2] + M.dg.zchunk - 1) / M.dg.zchunk;
      M.k7.ce = (float)h.params[0];
      M.k7.cw = (float)h.params[1];
      M.k7.cn = (float)h.params[2];
      M.k7.cs = (float)h.params[3];
      M.k7.ct = (float)h.params[4];
      M.k7.cb = (float)h.params[5];
      M.k7.cc = (float)h.params[6];
      PSB_CHECK(get_tmap(g0, M.dg.bx, M.dg.by, &a, kPromoD));
      PSB_CHECK(get_tmap(g1, M.dg.bx, M.dg.by, &c, kPromoD));
    }
    tmaps[2 * i] = *a;
    tmaps[2 * i + 1] = *c;
    M.ntiles = M.tiles_x * M.tiles_y * M.nzc;
    partial_slots += 2 * 2 * (group[i] == 2 ? kT2Units : kBWarps) * (int64_t)M.ntiles;
  }
  PSB_CHECK(dev_reserve(&b->d_tmaps, &b->cap_tmaps, sizeof(CUtensorMap) * tmaps.size()));
  PSB_TRY(cudaMemcpy(b->d_tmaps, tmaps.data(), sizeof(CUtensorMap) * tmaps.size(),
                     cudaMemcpyHostToDevice));
  PSB_CHECK(dev_reserve(&b->d_partials, &b->cap_partials,
                        sizeof(double) * std::max<int64_t>(1, partial_slots)));
  if (pass_words) {
    std::vector<int> flat;
    flat.reserve(pass_words);
    for (int i = 0; i < n; i++) flat.insert(flat.end(), b->passes[i].begin(), b->passes[i].end());
    PSB_CHECK(dev_reserve(&b->d_pass, &b->cap_pass, sizeof(int) * flat.size()));
    PSB_TRY(cudaMemcpy(b->d_pass, flat.data(), sizeof(int) * flat.size(), cudaMemcpyHostToDevice));
  }
  int64_t counters = 0;
  for (int i = 0; i < n; i++) counters += units[i] + b->members[i].ntiles;
  b->n_counters = std::max<int64_t>(1, counters);
  PSB_CHECK(dev_reserve(&b->d_done, &b->cap_done, sizeof(unsigned) * b->n_counters));
  PSB_CHECK(dev_reserve(&b->d_stop, &b->cap_stop, sizeof(int) * std::max(1, n)));
  PSB_CHECK(dev_reserve(&b->d_res, &b->cap_res, sizeof(double) * 4 * std::max(1, n)));
  if ((int)b->res_init.size() == 4 * n && n > 0)
    PSB_TRY(cudaMemcpy(b->d_res, b->res_init.data(), sizeof(double) * 4 * n, cudaMemcpyHostToDevice));
  else
    PSB_TRY(cudaMemset(b->d_res, 0, sizeof(double) * 4 * std::max(1, n)));
  int64_t off = 0, coff = 0, poff = 0;
  for (int i = 0; i < n; i++) {
    BMember &M = b->members[i];
    M.tmap[0] = b->d_tmaps + 2 * i;
    M.tmap[1] = b->d_tmaps + 2 * i + 1;
    M.tcoef = coef_map[i] >= 0 ? b->d_tmaps + coef_map[i] : nullptr;
    M.partials = b->d_partials + off;
    off += 2 * 2 * (group[i] == 2 ? kT2Units : kBWarps) * (int64_t)M.ntiles;
    M.step_cnt = b->d_done + coff;
    coff += units[i];
    M.tile_done = b->d_done + coff;
    coff += M.ntiles;
    M.stop = b->d_stop + i;
    M.res = b->d_res + 4 * i;
    if (group[i] == 2) {
      M.pass_start = b->d_pass + poff;
      poff += units[i] + 1;
    }
  }
  PSB_CHECK(dev_reserve(&b->d_members, &b->cap_members, sizeof(BMember) * std::max(1, n)));
  PSB_TRY(cudaMemcpy(b->d_members, b->members.data(), sizeof(BMember) * n, cudaMemcpyHostToDevice));
  // One work list per kernel kind, in units of steps (passes for group 2).
  // Members are ordered by units (descending), so the members still running
  // at unit s are a prefix.
  for (int gi = 0; gi < 3; gi++) {
    BatchGroup &G = b->grp[gi];
    G.order.clear();
    for (int i = 0; i < n; i++)
      if (group[i] == gi) G.order.push_back(i);
    std::stable_sort(G.order.begin(), G.order.end(),
                     [&](int x, int y) { return units[x] > units[y]; });
    const int gn = (int)G.order.size();
    G.tile_prefix.assign(gn + 1, 0);
    for (int i = 0; i < gn; i++)
      G.tile_prefix[i + 1] = G.tile_prefix[i] + b->members[G.order[i]].ntiles;
    G.max_steps = gn ? units[G.order[0]] : 0;
    G.step_offset.assign(G.max_steps + 1, 0);
    int active = gn;
    for (int st = 0; st < G.max_steps; st++) {
      while (active > 0 && units[G.order[active - 1]] <= st) active--;
      G.step_offset[st + 1] = G.step_offset[st] + G.tile_prefix[active];
    }
    G.total_items = G.max_steps ? G.step_offset[G.max_steps] : 0;
    G.work = 0;
    for (int i : G.order)
      G.work += (double)b->hm[i].points * steps[i] * (gi == 0 ? 8.0 : gi == 1 ? 56.0 : 28.0);
    PSB_CHECK(dev_reserve(&G.d_order, &G.cap_order, sizeof(int) * std::max(1, gn)));
    if (gn) PSB_TRY(cudaMemcpy(G.d_order, G.order.data(), sizeof(int) * gn, cudaMemcpyHostToDevice));
    PSB_CHECK(dev_reserve(&G.d_tile_prefix, &G.cap_tile_prefix, sizeof(int64_t) * (gn + 1)));
    PSB_TRY(cudaMemcpy(G.d_tile_prefix, G.tile_prefix.data(), sizeof(int64_t) * (gn + 1),
                       cudaMemcpyHostToDevice));
    PSB_CHECK(dev_reserve(&G.d_step_offset, &G.cap_step_offset,
                          sizeof(int64_t) * (G.max_steps + 1)));
    PSB_TRY(cudaMemcpy(G.d_step_offset, G.step_offset.data(), sizeof(int64_t) * (G.max_steps + 1),
                       cudaMemcpyHostToDevice));
    if (!G.d_cursor) PSB_TRY(device_malloc(&G.d_cursor, sizeof(unsigned long long)));
    int per_sm = 0;
    if (gi == 0) {
      PSB_TRY(cudaFuncSetAttribute(k_batch<0>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
      PSB_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<0>, kBThreads,
                                                            batch_smem(0)));
    } else if (gi == 1) {
      PSB_TRY(cudaFuncSetAttribute(k_batch<1>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
      PSB_TRY(cudaFuncSetAttribute(k_batch<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)batch_smem(1)));
      PSB_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<1>, kBThreads,
                                                            batch_smem(1)));
    } else {
      PSB_TRY(cudaFuncSetAttribute(k_batch_tb2, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)batch_smem(2)));
      PSB_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_tb2, kT2Threads,
                                                            batch_smem(2)));
    }
    G.blocks_persistent = std::max(1, per_sm) * r.sm_count;
  }
  b->built = true;
  return PSB_OK;
}

// Whether the steps of member i overlap as a wavefront in the prepared
// launch (the producer's per-tile dependency path).
bool batch_member_wavefront(const psb_batch *b, int i) {
  if (!b->built || i < 0 || i >= (int)b->members.size()) return false;
  const BMember &M = b->members[i];
  return M.ntiles >= kWaveTiles && (M.group == 2 ? M.npasses : M.steps) > 1;
}

int batch_member_cur(const psb_batch *b, int i, int done) {
  const BatchMemberHost &h = b->hm[i];
  if (!b->built || i >= (int)b->members.size() || b->members[i].group != 2)
    return (h.cur0 + done) & 1;
  // Passes that ended at or before `done` each flipped the buffer.
  const std::vector<int> &ps = b->passes[i];
  const int passes = (int)(std::upper_bound(ps.begin(), ps.end(), done) - ps.begin()) - 1;
  return (h.cur0 + passes) & 1;
}

// After a run: per member, local steps completed when it converged (-1 if
// it did not) and its residual state (4 doubles).
psb_status batch_read_state(psb_batch *b, std::vector<int> &stop, std::vector<double> &res) {
  const int n = (int)b->hm.size();
  stop.assign(n, -1);
  res.assign(4 * n, 0.0);
  if (!b->built || n == 0) return PSB_OK;
  PSB_TRY(cudaMemcpy(stop.data(), b->d_stop, sizeof(int) * n, cudaMemcpyDeviceToHost));
  PSB_TRY(cudaMemcpy(res.data(), b->d_res, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost));
  return PSB_OK;
}

psb_status batch_reset_counters(psb_batch *b, cudaStream_t s) {
  const int n = (int)b->hm.size();
  PSB_TRY(cudaMemsetAsync(b->d_done, 0, sizeof(unsigned) * b->n_counters, s));
  PSB_TRY(cudaMemsetAsync(b->d_stop, 0xff, sizeof(int) * std::max(1, n), s));
  for (auto &g : b->grp) PSB_TRY(cudaMemsetAsync(g.d_cursor, 0, sizeof(unsigned long long), s));
  return PSB_OK;
}

static BatchDev batch_dev(psb_batch *b, int gi) {
  const BatchGroup &G = b->grp[gi];
  BatchDev B;
  B.nmembers = (int)G.order.size();
  B.members = b->d_members;
  B.order = G.d_order;
  B.tile_prefix = G.d_tile_prefix;
  B.step_offset = G.d_step_offset;
  B.max_steps = G.max_steps;
  B.total_items = G.total_items;
  B.cursor = G.d_cursor;
  B.err = rt().d_error;
  return B;
}

static psb_status batch_side_stream(psb_batch *b) {
  if (!b->side) {
    PSB_TRY(cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking));
    PSB_TRY(cudaStreamCreateWithFlags(&b->side2, cudaStreamNonBlocking));
    PSB_TRY(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming));
    PSB_TRY(cudaEventCreateWithFlags(&b->join, cudaEventDisableTiming));
    PSB_TRY(cudaEventCreateWithFlags(&b->join2, cudaEventDisableTiming));
  }
  return PSB_OK;
}

// One launch of work list gi on stream ss (step < 0: persistent).
static psb_status batch_launch_group(psb_batch *b, int gi, cudaStream_t ss, int step,
                                     unsigned blocks) {
  const BatchDev B = batch_dev(b, gi);
  if (gi == 0)
    k_batch<0><<<blocks, kBThreads, batch_smem(0), ss>>>(B, step);
  else if (gi == 1)
    k_batch<1><<<blocks, kBThreads, batch_smem(1), ss>>>(B, step);
  else
    k_batch_tb2<<<blocks, kT2Threads, batch_smem(2), ss>>>(B, step);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e, "k_batch");
  return PSB_OK;
}

// Mode 0: the two kinds' persistent launches run concurrently, the one with
// more work launched first on `s`, the other on a side stream; the second
// launch's CTAs take slots as the first one's retire, so each fills the
// other's tail.
psb_status batch_launch_persistent(psb_batch *b, cudaStream_t s, int64_t *launches) {
  PSB_CHECK(batch_reset_counters(b, s));
  // Work lists with items, the one with most work first on s, the others on
  // side streams forked from s: each one's CTAs take slots as the others
  // retire, so they fill each other's tails.
  int order[3], nl = 0;
  for (int gi = 0; gi < 3; gi++)
    if (b->grp[gi].total_items) order[nl++] = gi;
  for (int i = 1; i < nl; i++)  // by work, descending (at most three lists)
    for (int j = i; j > 0 && b->grp[order[j]].work > b->grp[order[j - 1]].work; j--)
      std::swap(order[j], order[j - 1]);
  if (nl > 1) {
    PSB_CHECK(batch_side_stream(b));
    PSB_TRY(cudaEventRecord(b->fork, s));
    PSB_TRY(cudaStreamWaitEvent(b->side, b->fork, 0));
    if (nl > 2) PSB_TRY(cudaStreamWaitEvent(b->side2, b->fork, 0));
  }
  for (int k = 0; k < nl; k++) {
    const int gi = order[k];
    const BatchGroup &G = b->grp[gi];
    cudaStream_t ss = k == 0 ? s : (k == 1 ? b->side : b->side2);
    const int blocks = (int)std::min<int64_t>(G.blocks_persistent, G.total_items);
    PSB_CHECK(batch_launch_group(b, gi, ss, -1, (unsigned)blocks));
    (*launches)++;
  }
  if (nl > 1) {
    PSB_TRY(cudaEventRecord(b->join, b->side));
    PSB_TRY(cudaStreamWaitEvent(s, b->join, 0));
    if (nl > 2) {
      PSB_TRY(cudaEventRecord(b->join2, b->side2));
      PSB_TRY(cudaStreamWaitEvent(s, b->join2, 0));
    }
  }
  return PSB_OK;
}

// Per-step launches (mode 1): each work list's unit sequence (steps, or
// passes for two-sweep Himeno members) on its own stream, forked and joined
// inside one CUDA graph, recorded once and replayed.
psb_status batch_launch_graph(psb_batch *b, cudaStream_t s, int64_t *launches) {
  if (!b->graph) {
    PSB_CHECK(batch_side_stream(b));
    cudaGraph_t g;
    PSB_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    psb_status st = batch_reset_counters(b, s);
    cudaEventRecord(b->fork, s);
    cudaStreamWaitEvent(b->side, b->fork, 0);
    cudaStreamWaitEvent(b->side2, b->fork, 0);
    for (int gi = 0; gi < 3 && st == PSB_OK; gi++) {
      const BatchGroup &G = b->grp[gi];
      cudaStream_t ss = gi == 0 ? s : (gi == 1 ? b->side : b->side2);
      int active = (int)G.order.size();
      auto units = [&](int m) {
        const BMember &M = b->members[m];
        return M.group == 2 ? M.npasses : M.steps;
      };
      for (int step = 0; step < G.max_steps && st == PSB_OK; step++) {
        while (active > 0 && units(G.order[active - 1]) <= step) active--;
        st = batch_launch_group(b, gi, ss, step, (unsigned)G.tile_prefix[active]);
      }
    }
    cudaEventRecord(b->join, b->side);
    cudaStreamWaitEvent(s, b->join, 0);
    cudaEventRecord(b->join2, b->side2);
    cudaStreamWaitEvent(s, b->join2, 0);
    cudaError_t e = cudaStreamEndCapture(s, &g);
    if (st != PSB_OK || e != cudaSuccess) {
      if (e == cudaSuccess) cudaGraphDestroy(g);
      cudaGetLastError();
      return st != PSB_OK ? set_status(st) : cuda_status(e, "batch graph capture");
    }
    e = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_status(e, "batch graph instantiate");
  }
  PSB_TRY(cudaGraphLaunch(b->graph, s));
  *launches += b->grp[0].max_steps + b->grp[1].max_steps + b->grp[2].max_steps;
  return PSB_OK;
}

}  // namespace psb

// ===========================================================================
// C ABI
// ===========================================================================
namespace psb {

psb_batch *batch_new() {
  psb_batch *b = new psb_batch();
  cudaEventCreate(&b->ev0);
  cudaEventCreate(&b->ev1);
  return b;
}

void batch_set_members(psb_batch *b, const std::vector<BatchMemberHost> &m,
                       const std::vector<double> &res_init) {
  batch_invalidate(b);
  b->hm = m;
  b->res_init = res_init;
}

void batch_delete(psb_batch *b) {
  if (!b) return;
  batch_release_device(b);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->side) cudaStreamDestroy(b->side);
  if (b->side2) cudaStreamDestroy(b->side2);
  if (b->fork) cudaEventDestroy(b->fork);
  if (b->join) cudaEventDestroy(b->join);
  if (b->join2) cudaEventDestroy(b->join2);
  delete b;
}

psb_status batch_add_member(psb_batch *b, const BatchMemberHost &m) {
  b->hm.push_back(m);
  batch_invalidate(b);
  return PSB_OK;
}

// Per-grid loop (modes 2 and 3): each member alone with one launch per step.
static psb_status batch_run_loop(psb_batch *b, int impl, int64_t *launches) {
  Runtime &r = rt();
  const int old_impl = r.impl;
  const bool old_graph = r.use_graph;
  r.impl = impl;
  r.use_graph = impl != PSB_IMPL_PLAIN;  // the plain loop launches every step itself
  drop_all_graphs();
  psb_status st = PSB_OK;
  for (auto &h : b->hm) {
    __PSDomain dom = h.kind == BK_HIMENO
                         ? PSDomain3DNew(1, h.grids[0]->pub.dim[0] - 1, 1, h.grids[0]->pub.dim[1] - 1,
                                         1, h.grids[0]->pub.dim[2] - 1)
                         : PSDomain3DNew(0, h.grids[0]->pub.dim[0], 0, h.grids[0]->pub.dim[1], 0,
                                         h.grids[0]->pub.dim[2]);
    __PSGrid *fw[14], *bw[14];
    for (int i = 0; i < h.ngrids; i++) fw[i] = bw[i] = &h.grids[i]->pub;
    bw[0] = &h.grids[1]->pub;
    bw[1] = &h.grids[0]->pub;
    PSStencil m1 = 0, m2 = 0;
    st = psb_stencil_map(h.kernel_id, &dom, fw, h.ngrids, h.params, h.nparams, &m1);
    if (st == PSB_OK) st = psb_stencil_map(h.kernel_id, &dom, bw, h.ngrids, h.params, h.nparams, &m2);
    if (st == PSB_OK) {
      PSStencil ms[2] = {m1, m2};
      if (h.steps / 2) {
        st = psb_stencil_run(ms, 2, h.steps / 2);
        *launches += r.last_launches;
      }
      if (st == PSB_OK && (h.steps & 1)) {
        st = psb_stencil_run(ms, 1, 1);
        *launches += r.last_launches;
      }
    }
    if (m1) psb_stencil_free(m1);
    if (m2) psb_stencil_free(m2);
    if (st != PSB_OK) break;
  }
  r.impl = old_impl;
  r.use_graph = old_graph;
  drop_all_graphs();
  return st;
}

// Which members that would run two sweeps per item have different values around
// the domains of their two pressure grids now; a change ends the work lists built
// before. (The server's requests get the same values in both.)
static psb_status batch_check_rims(psb_batch *b) {
  std::vector<int> who, differ;
  for (int i = 0; i < (int)b->hm.size(); i++)
    if (two_sweep_member(b->hm[i], member_tune(b->hm[i]), b->hm[i].steps)) who.push_back(i);
  if (who.empty()) return PSB_OK;
  cudaStream_t s = rt().stream;
  differ.resize(who.size());
  const size_t bytes = sizeof(int) * who.size();
  PSB_CHECK(dev_reserve(&b->d_rims, &b->cap_rims, bytes));
  PSB_TRY(cudaMemsetAsync(b->d_rims, 0, bytes, s));
  for (size_t k = 0; k < who.size(); k++) {
    const BatchMemberHost &h = b->hm[who[k]];
    Dom3 d;
    for (int i = 0; i < 3; i++) {
      d.lo[i] = 1;
      d.hi[i] = h.grids[0]->pub.dim[i] - 1;
    }
    PSB_CHECK(himeno_rim_compare(h.grids[0], h.grids[1], d, b->d_rims + k, s));
  }
  PSB_TRY(cudaMemcpyAsync(differ.data(), b->d_rims, bytes, cudaMemcpyDeviceToHost, s));
  PSB_TRY(cudaStreamSynchronize(s));
  for (size_t k = 0; k < who.size(); k++) {
    bool &was = b->hm[who[k]].rims_differ;
    if (was == (differ[k] != 0)) continue;
    was = differ[k] != 0;
    batch_invalidate(b);
  }
  return PSB_OK;
}

}  // namespace psb

extern "C" {

psb_status psb_batch_create(psb_batch **b) {
  if (!b) return set_status(PSB_ERR_INVALID);
  PSB_CHECK(ensure_init());
  *b = new psb_batch();
  PSB_TRY(cudaEventCreate(&(*b)->ev0));
  PSB_TRY(cudaEventCreate(&(*b)->ev1));
  return PSB_OK;
}

psb_status psb_batch_add(psb_batch *b, int kernel_id, __PSGrid *const *grids, int ngrids,
                         const double *params, int nparams, int steps, int *member) {
  if (!b || !grids || steps < 0 || nparams < 0 || nparams > PSB_MAX_PARAMS)
    return set_status(PSB_ERR_INVALID);
  BatchMemberHost h;
  h.kernel_id = kernel_id;
  if (kernel_id == PSB_KERNEL_DIFFUSION7 || kernel_id == PSB_KERNEL_DIFFUSION7_PERIODIC) {
    if (ngrids != 2 || nparams != 7) return set_status(PSB_ERR_INVALID);
    h.kind = kernel_id == PSB_KERNEL_DIFFUSION7 ? BK_DIFF7 : BK_DIFF7P;
  } else if (kernel_id == PSB_KERNEL_HIMENO19) {
    if (ngrids != 14 || nparams != 1) return set_status(PSB_ERR_INVALID);
    h.kind = BK_HIMENO;
  } else {
    return set_status(PSB_ERR_UNSUPPORTED);
  }
  h.ngrids = ngrids;
  for (int i = 0; i < ngrids; i++) {
    GridImpl *g = as_impl(grids[i]);
    if (!g || g->layout != PSB_LAYOUT_PITCHED || g->type != PS_FLOAT || g->pub.num_dims != 3)
      return set_status(PSB_ERR_INVALID);
    for (int k = 0; k < 3; k++)
      if (g->pub.dim[k] != as_impl(grids[0])->pub.dim[k]) return set_status(PSB_ERR_INVALID);
    h.grids[i] = g;
  }
  if (h.grids[0] == h.grids[1]) return set_status(PSB_ERR_INVALID);
  const int *n = h.grids[0]->pub.dim;
  if (h.kind == BK_HIMENO && (n[0] < 3 || n[1] < 3 || n[2] < 3)) return set_status(PSB_ERR_INVALID);
  if (h.kind == BK_DIFF7P && (n[0] < PSB_HALO || n[1] < PSB_HALO || n[2] < PSB_HALO))
    return set_status(PSB_ERR_INVALID);
  for (int i = 0; i < nparams; i++) h.params[i] = params[i];
  h.nparams = nparams;
  h.steps = steps;
  h.points = h.kind == BK_HIMENO ? (int64_t)(n[0] - 2) * (n[1] - 2) * (n[2] - 2)
                                 : (int64_t)n[0] * n[1] * n[2];
  if (member) *member = (int)b->hm.size();
  return batch_add_member(b, h);
}

psb_status psb_batch_run(psb_batch *b, int mode) {
  if (!b) return set_status(PSB_ERR_INVALID);
  Runtime &r = rt();
  std::lock_guard<std::recursive_mutex> lk(r.mu);
  int64_t launches = 0;
  legacy_join_in();
  // Periodic members read their input's resident halo.
  for (auto &h : b->hm)
    if (h.kind == BK_DIFF7P && h.grids[0]->ghost_valid != PSB_BOUNDARY_PERIODIC &&
        h.grids[0]->ghost_valid != kGhostFaces)
      PSB_CHECK(launch_halo_fill(h.grids[0], PSB_BOUNDARY_PERIODIC, r.stream));
  if (mode == 0 || mode == 1) {
    PSB_CHECK(batch_check_rims(b));
    if (!b->built) {
      std::vector<int> steps, step0;
      for (auto &h : b->hm) {
        steps.push_back(h.steps);
        step0.push_back(0);
      }
      PSB_CHECK(batch_prepare(b, steps, step0));
    }
  }
  PSB_TRY(cudaEventRecord(b->ev0, r.stream));
  psb_status st;
  switch (mode) {
    case 0: st = batch_launch_persistent(b, r.stream, &launches); break;
    case 1: st = batch_launch_graph(b, r.stream, &launches); break;
    case 2: st = batch_run_loop(b, PSB_IMPL_PLAIN, &launches); break;
    case 3: st = batch_run_loop(b, PSB_IMPL_AUTO, &launches); break;
    default: return set_status(PSB_ERR_INVALID);
  }
  if (st != PSB_OK) return set_status(st);
  PSB_TRY(cudaEventRecord(b->ev1, r.stream));
  legacy_join_out();
  PSB_TRY(cudaEventSynchronize(b->ev1));
  float ms = 0;
  PSB_TRY(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
  b->last_ms = ms;
  b->last_launches = launches;
  int64_t lups = 0;
  for (auto &h : b->hm) {
    lups += h.points * h.steps;
    // Writers keep the output halo's faces of periodic members current.
    if (h.kind == BK_DIFF7P) {
      h.grids[0]->ghost_valid = kGhostFaces;
      h.grids[1]->ghost_valid = kGhostFaces;
    } else {
      h.grids[0]->ghost_valid = h.grids[1]->ghost_valid = PSB_BOUNDARY_NONE;
    }
  }
  b->last_lups = lups;
  int err = 0;
  PSB_TRY(cudaMemcpy(&err, r.d_error, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) {
    cudaMemset(r.d_error, 0, sizeof(int));
    return set_status(PSB_ERR_TIMEOUT);
  }
  return PSB_OK;
}

psb_status psb_batch_stats(psb_batch *b, double *device_ms, int64_t *launches,
                           int64_t *lattice_updates) {
  if (!b) return set_status(PSB_ERR_INVALID);
  if (device_ms) *device_ms = b->last_ms;
  if (launches) *launches = b->last_launches;
  if (lattice_updates) *lattice_updates = b->last_lups;
  return PSB_OK;
}

psb_status psb_batch_set_stop(psb_batch *b, int member, double tol, int check_every) {
  if (!b || member < 0 || member >= (int)b->hm.size() || tol < 0 || check_every < 0)
    return set_status(PSB_ERR_INVALID);
  b->hm[member].tol = tol;
  b->hm[member].check_every = check_every;
  batch_invalidate(b);
  return PSB_OK;
}

psb_status psb_batch_member_result(psb_batch *b, int member, int *steps_done, double *residual,
                                   int *result_grid) {
  if (!b || member < 0 || member >= (int)b->hm.size()) return set_status(PSB_ERR_INVALID);
  const BatchMemberHost &h = b->hm[member];
  int done = h.steps;
  double res = -1.0;
  if (b->built) {
    int stop = -1;
    double r4[4];
    PSB_TRY(cudaMemcpy(&stop, b->d_stop + member, sizeof(int), cudaMemcpyDeviceToHost));
    PSB_TRY(cudaMemcpy(r4, b->d_res + 4 * member, sizeof(r4), cudaMemcpyDeviceToHost));
    if (stop >= 0) done = stop;
    if (r4[3] > 0) res = r4[1] > 0 ? sqrt(r4[0] / r4[1]) : 0.0;
  }
  if (steps_done) *steps_done = done;
  if (residual) *residual = res;
  if (result_grid) *result_grid = batch_member_cur(b, member, done);
  return PSB_OK;
}

// Autotuner for batch members. For every size bucket (kind, element type,
// extents rounded up to powers of two) among the members that has no
// cached entry (or all of them, with force), a scratch member of the first
// member's extents runs alone in the persistent kernel for kTuneSteps
// steps under each candidate tile width and z chunk; the fastest (CUDA
// events, best of two runs after a warm-up) goes into the tune table and
// the cache file, where batch_prepare finds it for every member of that
// bucket. The reference's counterpart is its translation-time trial of
// optimisation variants (translator/reference_translator.cc:749-1223).
constexpr int kTuneSteps = 8;
// A fixed tile width or two sweeps per pass replaces the fewest-tiles rule
// only if its trial takes at most this fraction of the rule's time.
constexpr double kTuneMargin = 0.9;

// Bytes of scratch grids the tuner may hold at once for one bucket.
constexpr int64_t kTuneBytes = 4ll << 30;

static psb_status batch_tune_member(const BatchMemberHost &h, psb_tune_config *best_cfg) {
  Runtime &r = rt();
  const int ng = h.ngrids;
  const int *dim = h.grids[0]->pub.dim;
  const int rows_per_thread = h.kind == BK_HIMENO ? 1 : kVY;
  // Candidate 0 is the fewest-tiles rule itself, which every member of the
  // bucket applies to its own extents; a fixed width must beat it clearly,
  // since it is timed on one member's extents and then given to the whole
  // bucket.
  const std::vector<int> txs = {0, 8, 11, 16, 21, 32};
  const int nz = dim[2] - (h.kind == BK_HIMENO ? 2 : 0);
  // A member is timed the way it runs inside a full batch: enough identical
  // copies that one launch holds about two waves of items at the longest z
  // chunk (a lone small member would favour short chunks and narrow tiles
  // that a full batch does not need), within kTuneBytes of scratch grids.
  int tx_h = 0, ty_h = 0;
  pick_shape(dim[0], dim[1], rows_per_thread, &tx_h, &ty_h);
  const int64_t tiles64 = (int64_t)((dim[0] + tx_h * 4 - 1) / (tx_h * 4)) *
                          ((dim[1] + ty_h * rows_per_thread - 1) / (ty_h * rows_per_thread)) *
                          ((nz + 63) / 64);
  const int64_t grid_bytes = (int64_t)(h.grids[0]->alloc_bytes);
  int copies = (int)std::min<int64_t>(256, (2 * items_target() + tiles64 - 1) / tiles64);
  copies = (int)std::max<int64_t>(1, std::min<int64_t>(copies, kTuneBytes / (grid_bytes * ng)));
  std::vector<__PSGrid *> gs((size_t)ng * copies, nullptr);
  psb_status st = PSB_OK;
  for (size_t i = 0; i < gs.size() && st == PSB_OK; i++)
    st = psb_grid_new(PS_FLOAT, 3, dim, PSB_LAYOUT_PITCHED, &gs[i]);
  for (size_t i = 0; i < gs.size() && st == PSB_OK; i++) {
    const int f = (int)(i % ng);
    st = psb_grid_fill(gs[i], 0, 7 + f, h.kind == BK_HIMENO && f == 5 ? 0.15 : 0.0,
                       h.kind == BK_HIMENO && f == 5 ? 0.18 : 1.0);
  }
  psb_batch *tb = batch_new();
  std::vector<BatchMemberHost> ts(copies, h);
  for (int c = 0; c < copies; c++) {
    BatchMemberHost &t = ts[c];
    for (int i = 0; i < ng; i++) t.grids[i] = gs[(size_t)c * ng + i] ? as_impl(gs[(size_t)c * ng + i]) : nullptr;
    t.steps = kTuneSteps;
    t.check_every = 0;
    t.tol = 0;
    if (st == PSB_OK && h.kind == BK_DIFF7P)
      st = launch_halo_fill(t.grids[0], PSB_BOUNDARY_PERIODIC, r.stream);
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (st == PSB_OK && cudaEventCreate(&e0) != cudaSuccess) st = PSB_ERR_CUDA;
  if (st == PSB_OK && cudaEventCreate(&e1) != cudaSuccess) st = PSB_ERR_CUDA;
  double best = -1, rule_ms = -1;
  // The rule is the batch's default: the fewest-tiles shape with the
  // default sweeps per pass. Himeno buckets also try the other depth (two
  // sweeps: 64 x 12 tiles, recorded as tile_x 64).
  const int rule_td = h.kind == BK_HIMENO ? default_sweeps(h) : 1;
  std::vector<std::array<int, 2>> cands;  // (tile width in threads or 0, t_depth)
  cands.push_back({0, rule_td});
  for (int tx : txs)
    if (tx > 0) cands.push_back({tx, 1});
  if (h.kind == BK_HIMENO) cands.push_back(rule_td == 2 ? std::array<int, 2>{0, 1}
                                                        : std::array<int, 2>{kHtTX / 4, 2});
  // The z chunk is left to the batch's own rule (items per step over the
  // whole work list), as in a real run: a chunk that wins for the copies
  // alone is not the one a mixed batch would give this member.
  for (const auto &cd : cands) {
    const int tx = cd[0], td = cd[1];
    {
      if (st != PSB_OK) break;
      for (auto &t : ts) {
        t.force_tx = tx;
        t.force_zc = 0;
        t.force_td = td;
      }
      batch_set_members(tb, ts, {});
      st = batch_prepare(tb, std::vector<int>(copies, kTuneSteps), std::vector<int>(copies, 0));
      double ms_best = -1;
      for (int rep = 0; rep < 3 && st == PSB_OK; rep++) {
        int64_t launches = 0;
        cudaEventRecord(e0, r.stream);
        st = batch_launch_persistent(tb, r.stream, &launches);
        cudaEventRecord(e1, r.stream);
        if (st == PSB_OK && cudaEventSynchronize(e1) != cudaSuccess) st = PSB_ERR_CUDA;
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0 && (ms_best < 0 || ms < ms_best)) ms_best = ms;  // rep 0 warms up
      }
      if (__ps_trace)
        fprintf(__ps_trace, "physis_b200: batch tune kind=%d tile=%dx%d t=%d: %.4f ms\n",
                h.kind, tx * 4, td == 2 ? kHtTY : tx ? (kBConsumers / tx) * rows_per_thread : 0,
                td, ms_best);
      const bool rule = tx == 0 && td == rule_td;
      if (rule) rule_ms = ms_best;
      const double bar = rule ? best : std::min(best, kTuneMargin * rule_ms);
      if (st == PSB_OK && ms_best > 0 && (best < 0 || ms_best < bar)) {
        best = ms_best;
        best_cfg->impl = PSB_IMPL_TMA;
        best_cfg->tile_x = tx * 4;  // 0: the fewest-tiles rule
        best_cfg->tile_y = td == 2 ? kHtTY : tx ? (kBConsumers / tx) * rows_per_thread : 0;
        best_cfg->z_chunk = 0;  // the batch's rule
        best_cfg->stages = kBStages;
        best_cfg->t_depth = td;
      }
    }
  }
  batch_delete(tb);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  for (auto g : gs)
    if (g) PSGridFree(g);
  int err = 0;
  cudaMemcpy(&err, r.d_error, sizeof(int), cudaMemcpyDeviceToHost);
  if (err) {
    cudaMemset(r.d_error, 0, sizeof(int));
    return set_status(PSB_ERR_TIMEOUT);
  }
  if (st == PSB_OK && best < 0) st = PSB_ERR_UNSUPPORTED;
  return st;
}

psb_status psb_batch_autotune(psb_batch *b, int force) {
  if (!b) return set_status(PSB_ERR_INVALID);
  PSB_CHECK(ensure_init());
  Runtime &r = rt();
  std::lock_guard<std::recursive_mutex> lk(r.mu);
  legacy_join_in();
  PSB_TRY(cudaStreamSynchronize(r.stream));
  std::vector<std::array<int, 4>> done;
  bool stored = false;
  for (auto &h : b->hm) {
    int bucket[3];
    batch_tune_bucket(h.grids[0]->pub.dim, bucket);
    std::array<int, 4> key = {h.kind, bucket[0], bucket[1], bucket[2]};
    if (std::find(done.begin(), done.end(), key) != done.end()) continue;
    done.push_back(key);
    psb_tune_config cfg;
    if (!force && batch_tune_find(h.kind, h.grids[0]->pub.dim, &cfg)) continue;
    PSB_CHECK(batch_tune_member(h, &cfg));
    batch_tune_store(h.kind, h.grids[0]->pub.dim, cfg);
    stored = true;
  }
  if (stored) tune_save();
  batch_invalidate(b);
  return PSB_OK;
}

psb_status psb_batch_member_layout(psb_batch *b, int member, psb_batch_layout *layout) {
  if (!b || !layout || member < 0 || member >= (int)b->hm.size() || !b->built)
    return set_status(PSB_ERR_INVALID);
  const BMember &M = b->members[member];
  const bool him = M.kind == BK_HIMENO;
  layout->tile_x = M.group == 2 ? kHtTX : (him ? M.hg.tx_threads : M.dg.tx_threads) * 4;
  layout->tile_y = M.group == 2 ? kHtTY : him ? M.hg.ty_threads : M.dg.ty_threads * kVY;
  layout->z_chunk = him ? M.hg.zchunk : M.dg.zchunk;
  layout->tiles = M.ntiles;
  layout->wavefront = batch_member_wavefront(b, member) ? 1 : 0;
  const MemberTune mt = member_tune(b->hm[member]);
  layout->tuned = mt.tuned ? 1 : 0;
  layout->t_depth = M.group == 2 ? 2 : 1;
  layout->units = M.group == 2 ? M.npasses : M.steps;
  return PSB_OK;
}

psb_status psb_batch_free(psb_batch *b) {
  if (!b) return set_status(PSB_ERR_INVALID);
  cudaStreamSynchronize(rt().stream);
  batch_release_device(b);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->side) cudaStreamDestroy(b->side);
  if (b->side2) cudaStreamDestroy(b->side2);
  if (b->fork) cudaEventDestroy(b->fork);
  if (b->join) cudaEventDestroy(b->join);
  if (b->join2) cudaEventDestroy(b->join2);
  delete b;
  return PSB_OK;
}

}  // extern "C"
