// FP64 reduction accumulators shared by the grid reduction (k_reduce.cu)
// and the kernel-function reduction (k_generic.cu): SUM with Neumaier
// compensation, PROD in FP64, MAX/MIN exact; fixed shuffle trees, one
// partial per CTA, combined by the last CTA in index order.
#pragma once

#include <cfloat>

#include "device.cuh"

namespace psb {

constexpr int kReduceMaxBlocks = 1184;  // 148 SMs x 8: capacity of the partials

struct RAcc {
  double s;  // value (sum, product, max or min)
  double c;  // compensation (SUM only)
};

__host__ __device__ __forceinline__ RAcc racc_init(int op) {
  RAcc a;
  a.c = 0.0;
  switch (op) {
    case PS_MAX: a.s = -DBL_MAX; break;
    case PS_MIN: a.s = DBL_MAX; break;
    case PS_SUM: a.s = 0.0; break;
    default: a.s = 1.0; break;
  }
  return a;
}

// Neumaier step: add x to (s, c).
__host__ __device__ __forceinline__ void neumaier(RAcc &a, double x) {
  double t = a.s + x;
  if (fabs(a.s) >= fabs(x)) a.c += (a.s - t) + x;
  else a.c += (x - t) + a.s;
  a.s = t;
}

__host__ __device__ __forceinline__ RAcc racc_merge(int op, RAcc a, RAcc b) {
  switch (op) {
    case PS_MAX: a.s = a.s > b.s ? a.s : b.s; return a;
    case PS_MIN: a.s = a.s < b.s ? a.s : b.s; return a;
    case PS_SUM: {
      RAcc r = a;
      neumaier(r, b.s);
      r.c += b.c;
      return r;
    }
    default: a.s = a.s * b.s; return a;
  }
}

__host__ __device__ __forceinline__ void racc_add(int op, RAcc &a, double x) {
  switch (op) {
    case PS_MAX: a.s = a.s > x ? a.s : x; break;
    case PS_MIN: a.s = a.s < x ? a.s : x; break;
    case PS_SUM: neumaier(a, x); break;
    default: a.s = a.s * x; break;
  }
}

// Elements of a segment per thread: loads in flight (1 KB a warp).
template <typename T>
constexpr int kReduceU = 32 / (int)sizeof(T);
constexpr int kReduceAcc = 4;  // accumulators per thread

// One thread's share of a domain of rx x ry x rz elements from `base`: lane
// `lane` of the segments of warp `warp` of `nwarps`. (Host code runs it in the
// tests.)
template <typename T, int OP>
__host__ __device__ __forceinline__ RAcc reduce_thread(const T *base, int64_t sy, int64_t sz,
                                                       int rx, int ry, int rz, int64_t warp,
                                                       int64_t nwarps, int lane) {
  constexpr int U = kReduceU<T>;
  static_assert(U % kReduceAcc == 0, "every accumulator takes the same number of elements");
  const int segs = (int)(((int64_t)rx + 32 * U - 1) / (32 * U));
  // This warp's segments, `nwarps` apart in (z, y, segment) order, advanced
  // by carries (64-bit: a row may be up to 2^31-1 elements long).
  const int64_t drow = nwarps / segs, row0 = warp / segs;
  const int ds = (int)(nwarps % segs), dy = (int)(drow % ry);
  const int64_t dz = drow / ry;
  int s = (int)(warp % segs), y = (int)(row0 % ry);
  int64_t z = row0 / ry;
  RAcc a[kReduceAcc];
#pragma unroll
  for (int u = 0; u < kReduceAcc; u++) a[u] = racc_init(OP);
  while (z < rz) {
    const T *row = base + y * sy + z * sz;
    const int64_t x0 = (int64_t)s * (32 * U) + lane;
    T v[U];
    if (x0 - lane + 32 * U <= rx) {
#pragma unroll
      for (int u = 0; u < U; u++) v[u] = row[x0 + 32 * u];
#pragma unroll
      for (int u = 0; u < U; u++) racc_add(OP, a[u % kReduceAcc], (double)v[u]);
    } else {
#pragma unroll
      for (int u = 0; u < U; u++)
        if (x0 + 32 * u < rx) racc_add(OP, a[u % kReduceAcc], (double)row[x0 + 32 * u]);
    }
    s += ds;
    int cy = 0;
    if (s >= segs) {
      s -= segs;
      cy = 1;
    }
    // y + dy + cy may exceed 2^31 - 1 before the carry.
    int64_t y2 = (int64_t)y + dy + cy;
    z += dz;
    if (y2 >= ry) {
      y2 -= ry;
      z++;
    }
    y = (int)y2;
  }
#pragma unroll
  for (int u = 1; u < kReduceAcc; u++) a[0] = racc_merge(OP, a[0], a[u]);
  return a[0];
}

__device__ __forceinline__ RAcc racc_block(int op, RAcc v, RAcc *scratch) {
  for (int o = 16; o > 0; o >>= 1) {
    RAcc u;
    u.s = __shfl_down_sync(0xffffffffu, v.s, o);
    u.c = __shfl_down_sync(0xffffffffu, v.c, o);
    v = racc_merge(op, v, u);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  RAcc r = racc_init(op);
  if (warp == 0) {
    if (lane < nw) r = scratch[lane];
    for (int o = 16; o > 0; o >>= 1) {
      RAcc u;
      u.s = __shfl_down_sync(0xffffffffu, r.s, o);
      u.c = __shfl_down_sync(0xffffffffu, r.c, o);
      r = racc_merge(op, r, u);
    }
  }
  return r;
}

struct ReduceScratch {
  RAcc *partials;
  unsigned *ticket;
  double *result;
};

// The runtime-owned partials / ticket / result buffer (allocated once).
psb_status reduce_scratch(ReduceScratch *sc);

}  // namespace psb
