// Himeno two-sweep tile machinery (temporal blocking of depth 2), shared by
// the single-grid pass (k_himeno_tb2.cu) and the batched kernel (batch.cu).
//
// One tile of TX x TY points over a z chunk advances two sweeps. Rings
// (all in one CTA's shared memory, positions carried from tile to tile):
//  R1  input pressure planes, box TX+8 x TY+4 (the tile with a 2-cell halo,
//      x from x0-4 so the box starts on 16 bytes); one producer arrival,
//      one release per stage-1 and edge warp;
//  RC  the twelve coefficient boxes of a plane, TX+8 x TY+2 (a 1-cell
//      halo), field f at f * kHtField; one producer arrival, one release
//      per stage-1, edge and stage-2 warp;
//  R2  first-sweep planes over the tile and its 1-cell halo, laid out like
//      one coefficient box; one arrival per stage-1 and edge warp, one
//      release per stage-2 warp.
// Stage 1 (7 warps) and the edge warp compute the first sweep over (TX+2) x
// (TY+2) points per plane: stage 1 the 64-point rows as float4 vectors, the
// edge warp the two halo columns, 28 scalar points; points outside the domain
// take the value that the grid written by the first sweep holds there (HtRim),
// or the input's where they are known to be the same. Stage 2 (6
// warps) computes the second sweep of the tile from R2 and stores it, or (copy)
// stores the first sweep itself, which makes a one-sweep pass of the same
// rings. Both use the single-sweep arithmetic (himeno_point), so results equal
// single sweeps bit for bit.
//
// What bounds it: one CTA fits an SM, so loads and warps in flight are scarce.
// Every warp holds the planes around its points in registers and reads each
// plane and coefficient stage once, first thing in the turn, and releases it
// there: the rings are then prefetch only, and shared memory carries 84
// wavefronts per warp and plane instead of 124. The halo columns have a warp of
// their own (as lanes of the stage-1 warps they added a point's chain to the
// slower stage), and what shared memory the rings gave up went into twelve rows
// per tile, which read 1.17 coefficient rows per row instead of 1.25.
// 257 x 257 x 513, us per sweep: 272 with eight rows and planes read from the
// rings; 253 with the edge warp; 232 with the planes in registers; 208 released
// early, 202 with five coefficient stages; 184 with twelve rows (0.78 of the
// measured peak for the pass's 28 B per update). It spills 68 bytes a thread, at
// 128 registers. Fourteen rows need 17 warps, which leave 96 registers, and spill
// far more (458); two points a thread instead of four changes nothing; x
// neighbours by shuffle cost 8% (a longer chain).
#pragma once

#include "k_himeno.cuh"

namespace psb {

constexpr int kHtTX = 64, kHtTY = 12, kHtV = 4;
constexpr int kHtBX = kHtTX + 8;           // every box: x from x0 - 4
constexpr int kHtBY1 = kHtTY + 4;          // input p: y from y0 - 2
constexpr int kHtBY2 = kHtTY + 2;          // first sweep and coefficients: y from y0 - 1
// Ring depths (stages) of R1, R2 and RC; build options for measurement.
#ifndef PSB_HT_S1
#define PSB_HT_S1 4
#endif
#ifndef PSB_HT_S2
#define PSB_HT_S2 3
#endif
#ifndef PSB_HT_SC
#define PSB_HT_SC 4
#endif
constexpr int kHtS1 = PSB_HT_S1, kHtS2 = PSB_HT_S2, kHtSC = PSB_HT_SC;
static_assert(kHtS1 <= 8 && kHtS2 <= 8 && kHtSC <= 8, "eight barrier slots per ring");
constexpr int kHtStage1 = (kHtBX * kHtBY1 * 4 + 127) / 128 * 128;
constexpr int kHtStage2 = (kHtBX * kHtBY2 * 4 + 127) / 128 * 128;
constexpr int kHtField = kHtStage2;        // one coefficient box
constexpr int kHtStageC = 12 * kHtField;
constexpr int kHtW1 = kHtTX / kHtV * (kHtTY + 2) / 32;  // stage-1 warps
constexpr int kHtW2 = kHtTX / kHtV * kHtTY / 32;        // stage-2 warps; one edge warp more
constexpr int kHtEdge = 2 * (kHtTY + 2);   // points of the two halo columns
constexpr int kHtRingBytes = kHtS1 * kHtStage1 + kHtS2 * kHtStage2 + kHtSC * kHtStageC;
static_assert(kHtTX / kHtV * (kHtTY + 2) == 32 * kHtW1, "stage-1 threads cover the halo rows");
static_assert(kHtTX / kHtV * kHtTY == 32 * kHtW2, "stage-2 threads cover the tile");
static_assert(kHtEdge <= 32, "one edge point per lane");

struct HtRings {
  uint64_t *f1, *e1, *f2, *e2, *fc, *ec;  // full/empty barriers (8 slots each)
  unsigned char *r1, *r2, *rc;
};

// Barriers at bars[0..48) and rings from `rings` (kHtRingBytes).
__device__ __forceinline__ HtRings ht_rings(uint64_t *bars, unsigned char *rings) {
  HtRings R;
  R.f1 = bars;
  R.e1 = bars + 8;
  R.f2 = bars + 16;
  R.e2 = bars + 24;
  R.fc = bars + 32;
  R.ec = bars + 40;
  R.r1 = rings;
  R.r2 = R.r1 + kHtS1 * kHtStage1;
  R.rc = R.r2 + kHtS2 * kHtStage2;
  return R;
}

__device__ __forceinline__ void ht_init(const HtRings &R) {
  for (int i = 0; i < kHtS1; i++) {
    mbar_init(&R.f1[i], 1);
    mbar_init(&R.e1[i], kHtW1 + 1);
  }
  for (int i = 0; i < kHtS2; i++) {
    mbar_init(&R.f2[i], kHtW1 + 1);
    mbar_init(&R.e2[i], kHtW2);
  }
  for (int i = 0; i < kHtSC; i++) {
    mbar_init(&R.fc[i], 1);
    mbar_init(&R.ec[i], kHtW1 + 1 + kHtW2);
  }
}

__device__ __forceinline__ bool ht_wait(uint64_t *bar, uint32_t parity) {
  const bool ok = mbar_wait_bounded(bar, parity);
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void ht_release(uint64_t *bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// Producer (one thread): input planes zb-2 .. zb+nzl+1 into R1 and
// coefficient planes zb-1 .. zb+nzl into RC, each RC plane issued after the
// R1 plane the first sweep needs with it, so neither ring waits on a stage
// of the other that is not yet issued. coef: 12 tensor maps, one per field.
// (ax0, ay0, az0): tensor coordinates of logical (0,0,0). False if a
// bounded wait gave up.
__device__ __forceinline__ bool ht_produce_tile(const HtRings &R, RingPos &p1, RingPos &pc,
                                                const CUtensorMap *tin, const CUtensorMap *coef,
                                                int ax0, int ay0, int az0, int x0, int y0,
                                                int zb, int nzl) {
  auto put1 = [&](int z) -> bool {
    if (p1.round > 0 && !mbar_wait_bounded(&R.e1[p1.slot], (p1.round - 1) & 1)) return false;
    mbar_arrive_expect_tx(&R.f1[p1.slot], (uint32_t)(kHtBX * kHtBY1 * 4));
    tma_load_3d(R.r1 + p1.slot * kHtStage1, tin, &R.f1[p1.slot], x0 - 4 + ax0, y0 - 2 + ay0,
                z + az0);
    ring_next(p1, kHtS1);
    return true;
  };
  auto putc = [&](int z) -> bool {
    if (pc.round > 0 && !mbar_wait_bounded(&R.ec[pc.slot], (pc.round - 1) & 1)) return false;
    mbar_arrive_expect_tx(&R.fc[pc.slot], (uint32_t)(12 * kHtBX * kHtBY2 * 4));
    unsigned char *dst = R.rc + pc.slot * kHtStageC;
    for (int f = 0; f < 12; f++)
      tma_load_3d(dst + f * kHtField, coef + f, &R.fc[pc.slot], x0 - 4 + ax0, y0 - 1 + ay0,
                  z + az0);
    ring_next(pc, kHtSC);
    return true;
  };
  if (!put1(zb - 2) || !put1(zb - 1)) return false;
  for (int j = 0; j < nzl + 2; j++)
    if (!put1(zb + j) || !putc(zb - 1 + j)) return false;
  return true;
}

// After a producer gave up: wait (bounded) for its copies in flight.
__device__ __forceinline__ void ht_drain(const HtRings &R, RingPos p1, RingPos pc) {
  ring_drain(Ring{R.f1, R.e1, R.r1, kHtS1, kHtStage1}, p1);
  ring_drain(Ring{R.fc, R.ec, R.rc, kHtSC, kHtStageC}, pc);
}

// The walk's first two planes, each released as soon as it is in registers.
template <int V>
__device__ __forceinline__ bool ht_begin(HimenoWalk<V> &h, RingPos &p, int S, uint64_t *full,
                                         uint64_t *empty, const unsigned char *ring, int stage,
                                         int ofs, int lane) {
#pragma unroll
  for (int i = 0; i < 2; i++) {
    if (!ht_wait(&full[p.slot], p.round & 1)) return false;
    h.step();
    h.load(reinterpret_cast<const float *>(ring + p.slot * stage), ofs, kHtBX);
    ht_release(&empty[p.slot], lane);
    ring_next(p, S);
  }
  return true;
}

// The grid that the first sweep writes. Its values outside the domain are the
// first sweep's there, as a sweep leaves them (p: logical (0,0,0); nx, ny:
// points inside the grid). mid: p where the first sweep's own values are to be
// stored too (a run's last pass), else null.
struct HtRim {
  const float *p;
  int64_t sy, sz;
  int nx, ny;
  float *mid;
};

// Stage-1 warps (thread t in [0, 224)): the first sweep of one tile into R2.
// Thread t owns 4 x points of halo row t / 16 (y = y0 - 1 + row). Points
// outside the domain take their value from rim (RIM; fetched to L1 at the head
// of the turn, read at its end) or keep the input's. The two mostly are the same
// and the loads cost 10 to 40%, so the caller chooses. With acc_on, the FP64 sum of
// ss*ss over the tile's own domain points is added to *acc. False
// (warp-uniformly) if a bounded wait gave up.
template <bool RIM>
__device__ __forceinline__ bool ht_stage1_tile(const HtRings &R, RingPos &p1, RingPos &pc,
                                               RingPos &p2, int t, int lane, const Dom3 d,
                                               float omega, int x0, int y0, int zb, int nzl,
                                               bool acc_on, double *acc,
                                               const HtRim rim = HtRim{}) {
  const int tx = t % (kHtTX / kHtV), row = t / (kHtTX / kHtV);
  const int cofs = row * kHtBX + 4 + tx * kHtV;        // R2 / RC offset of the vector
  const int pofs = (row + 1) * kHtBX + 4 + tx * kHtV;  // R1 offset of the vector
  const int xg = x0 + tx * kHtV, yg = y0 - 1 + row;
  const bool row_in = yg >= d.lo[1] && yg < d.hi[1];
  const bool row_own = row_in && row >= 1 && row <= kHtTY;
  const bool xy_in = row_in && xg >= d.lo[0] && xg + kHtV <= d.hi[0];
  // The vector's points in the rim grid (a row of a pitched grid ends on a
  // whole vector).
  const bool has_rim = RIM && xg < rim.nx && yg < rim.ny;
  auto rim_at = [&](int z) { return rim.p + xg + (int64_t)yg * rim.sy + (int64_t)z * rim.sz; };
  HimenoWalk<kHtV> h = {};
  if (!ht_begin(h, p1, kHtS1, R.f1, R.e1, R.r1, kHtStage1, pofs, lane)) return false;
  double a = 0.0;
  for (int j = 0; j < nzl + 2; j++) {
    const int z = zb - 1 + j;
    const bool z_in = z >= d.lo[2] && z < d.hi[2];
    if (has_rim && !(z_in && xy_in))
      asm volatile("prefetch.global.L1 [%0];" ::"l"(rim_at(z)));
    if (!ht_wait(&R.f1[p1.slot], p1.round & 1) || !ht_wait(&R.fc[pc.slot], pc.round & 1))
      return false;
    const unsigned char *cs = R.rc + pc.slot * kHtStageC;
    Vec16<float> co[12];
#pragma unroll
    for (int f = 0; f < 12; f++)
      co[f] = lds16(reinterpret_cast<const float *>(cs + f * kHtField) + cofs);
    h.step();
    h.load(reinterpret_cast<const float *>(R.r1 + p1.slot * kHtStage1), pofs, kHtBX);
    ht_release(&R.e1[p1.slot], lane);
    ht_release(&R.ec[pc.slot], lane);  // stage 2 holds its own claim on the stage
    ring_next(p1, kHtS1);
    ring_next(pc, kHtSC);
    const bool z_own = z_in && j >= 1 && j <= nzl;
    float outv[kHtV];
#pragma unroll
    for (int v = 0; v < kHtV; v++) {
      const int x = xg + v;
      float c[12];
#pragma unroll
      for (int f = 0; f < 12; f++) c[f] = co[f].v[v];
      float ss;
      const float r = h.point(c, v, omega, &ss);
      const bool in = z_in && row_in && x >= d.lo[0] && x < d.hi[0];
      outv[v] = in || RIM ? r : h.c[1 + v];
      if (acc_on && in && z_own && row_own) a += (double)ss * (double)ss;
    }
    if (has_rim && !(z_in && xy_in)) {
      const float4 q = __ldg(reinterpret_cast<const float4 *>(rim_at(z)));
      const float w[kHtV] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int v = 0; v < kHtV; v++)
        if (!(z_in && row_in && xg + v >= d.lo[0] && xg + v < d.hi[0])) outv[v] = w[v];
    }
    if (rim.mid && z_own && row_own) {
      float *q = rim.mid + xg + (int64_t)yg * rim.sy + (int64_t)z * rim.sz;
      if (xy_in) {
        *reinterpret_cast<float4 *>(q) = make_float4(outv[0], outv[1], outv[2], outv[3]);
      } else {
#pragma unroll
        for (int v = 0; v < kHtV; v++)
          if (xg + v >= d.lo[0] && xg + v < d.hi[0]) q[v] = outv[v];
      }
    }
    // The first-sweep plane z into the next stage of R2.
    if (p2.round > 0 && !ht_wait(&R.e2[p2.slot], (p2.round - 1) & 1)) return false;
    float *dst = reinterpret_cast<float *>(R.r2 + p2.slot * kHtStage2);
    *reinterpret_cast<float4 *>(dst + cofs) = make_float4(outv[0], outv[1], outv[2], outv[3]);
    ht_release(&R.f2[p2.slot], lane);
    ring_next(p2, kHtS2);
  }
  *acc += a;
  return true;
}

// The edge warp: the first sweep's halo columns x0 - 1 and x0 + TX of one
// tile into R2, lane e < 28 the point of row e % 14 of column e / 14; rim as in
// stage 1. False (warp-uniformly) if a bounded wait gave up.
template <bool RIM>
__device__ __forceinline__ bool ht_edge_tile(const HtRings &R, RingPos &p1, RingPos &pc,
                                             RingPos &p2, int lane, const Dom3 d, float omega,
                                             int x0, int y0, int zb, int nzl,
                                             const HtRim rim = HtRim{}) {
  const int e = min(lane, kHtEdge - 1);
  const int col = e / (kHtTY + 2), row = e % (kHtTY + 2);
  const int xo = col ? 4 + kHtTX : 3;
  const int cofs = row * kHtBX + xo, pofs = (row + 1) * kHtBX + xo;
  const int x = col ? x0 + kHtTX : x0 - 1, y = y0 - 1 + row;
  const bool in_xy = y >= d.lo[1] && y < d.hi[1] && x >= d.lo[0] && x < d.hi[0];
  const float *rp = nullptr;
  if (RIM && x >= 0 && x < rim.nx && y < rim.ny)
    rp = rim.p + x + (int64_t)y * rim.sy + (int64_t)(zb - 1) * rim.sz;
  HimenoWalk<1> h = {};
  if (!ht_begin(h, p1, kHtS1, R.f1, R.e1, R.r1, kHtStage1, pofs, lane)) return false;
  for (int j = 0; j < nzl + 2; j++) {
    const int z = zb - 1 + j;
    const bool in = in_xy && z >= d.lo[2] && z < d.hi[2];
    float rv = 0.f;
    if (RIM) {
      if (!in && rp) rv = __ldg(rp);
      if (rp) rp += rim.sz;
    }
    if (!ht_wait(&R.f1[p1.slot], p1.round & 1) || !ht_wait(&R.fc[pc.slot], pc.round & 1))
      return false;
    const unsigned char *cs = R.rc + pc.slot * kHtStageC;
    float c[12];
#pragma unroll
    for (int f = 0; f < 12; f++) c[f] = reinterpret_cast<const float *>(cs + f * kHtField)[cofs];
    h.step();
    h.load(reinterpret_cast<const float *>(R.r1 + p1.slot * kHtStage1), pofs, kHtBX);
    ht_release(&R.e1[p1.slot], lane);
    ht_release(&R.ec[pc.slot], lane);
    ring_next(p1, kHtS1);
    ring_next(pc, kHtSC);
    float ss;
    const float r = h.point(c, 0, omega, &ss);
    const float out = in ? r : RIM ? rv : h.c[1];
    if (p2.round > 0 && !ht_wait(&R.e2[p2.slot], (p2.round - 1) & 1)) return false;
    if (lane < kHtEdge) reinterpret_cast<float *>(R.r2 + p2.slot * kHtStage2)[cofs] = out;
    ht_release(&R.f2[p2.slot], lane);
    ring_next(p2, kHtS2);
  }
  return true;
}

// Stage-2 warps (thread t in [0, 192)): the second sweep of the tile from R2
// and the coefficient stages of its planes, stored to pout (copy: the first
// sweep itself is stored). Thread t owns 4 x points of tile row t / 16.
// With acc_on (and not copy), the FP64 sum of ss*ss over the tile's domain
// points is added to *acc. False (warp-uniformly) if a bounded wait gave up.
__device__ __forceinline__ bool ht_stage2_tile(const HtRings &R, RingPos &p2, RingPos &pc, int t,
                                               int lane, float *pout, int64_t sy, int64_t sz,
                                               const Dom3 d, float omega, int x0, int y0,
                                               int zb, int nzl, bool copy, bool acc_on,
                                               double *acc) {
  const int tx = t % (kHtTX / kHtV), row = t / (kHtTX / kHtV);
  const int ofs = (row + 1) * kHtBX + 4 + tx * kHtV;
  const int xg = x0 + tx * kHtV, yg = y0 + row;
  const bool row_in = yg >= d.lo[1] && yg < d.hi[1];
  const bool xvec = xg >= d.lo[0] && xg + kHtV <= d.hi[0];
  // Coefficient plane zb-1 (the first sweep's near halo plane) is not read.
  if (!ht_wait(&R.fc[pc.slot], pc.round & 1)) return false;
  ht_release(&R.ec[pc.slot], lane);
  ring_next(pc, kHtSC);
  HimenoWalk<kHtV> h = {};
  if (!ht_begin(h, p2, kHtS2, R.f2, R.e2, R.r2, kHtStage2, ofs, lane)) return false;
  double a = 0.0;
  int64_t off = (int64_t)xg + (int64_t)yg * sy + (int64_t)zb * sz;
  for (int i = 0; i < nzl; i++) {
    // The coefficients are there before the first-sweep plane z+1 is.
    if (!ht_wait(&R.fc[pc.slot], pc.round & 1)) return false;
    const unsigned char *cs = R.rc + pc.slot * kHtStageC;
    Vec16<float> co[12];
#pragma unroll
    for (int f = 0; f < 12; f++)
      co[f] = lds16(reinterpret_cast<const float *>(cs + f * kHtField) + ofs);
    ht_release(&R.ec[pc.slot], lane);
    ring_next(pc, kHtSC);
    if (!ht_wait(&R.f2[p2.slot], p2.round & 1)) return false;
    h.step();
    h.load(reinterpret_cast<const float *>(R.r2 + p2.slot * kHtStage2), ofs, kHtBX);
    ht_release(&R.e2[p2.slot], lane);
    ring_next(p2, kHtS2);
    if (row_in) {
      float outv[kHtV];
#pragma unroll
      for (int v = 0; v < kHtV; v++) {
        float c[12];
#pragma unroll
        for (int f = 0; f < 12; f++) c[f] = co[f].v[v];
        float ss;
        const float r = h.point(c, v, omega, &ss);
        outv[v] = copy ? h.c[1 + v] : r;
        if (acc_on && !copy && xg + v >= d.lo[0] && xg + v < d.hi[0])
          a += (double)ss * (double)ss;
      }
      float *dst = pout + off;
      if (xvec) {
        *reinterpret_cast<float4 *>(dst) = make_float4(outv[0], outv[1], outv[2], outv[3]);
      } else {
#pragma unroll
        for (int v = 0; v < kHtV; v++)
          if (xg + v >= d.lo[0] && xg + v < d.hi[0]) dst[v] = outv[v];
      }
    }
    off += sz;
  }
  // Coefficient plane zb+nzl (the first sweep's far halo plane).
  if (!ht_wait(&R.fc[pc.slot], pc.round & 1)) return false;
  ht_release(&R.ec[pc.slot], lane);
  ring_next(pc, kHtSC);
  *acc += a;
  return true;
}

}  // namespace psb
