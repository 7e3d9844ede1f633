// Device side of the compiled point kernel of a generic stencil
// (k_generic_pt.cu writes the kernel's source for one table). Included by
// that source, so it compiles under the run-time compiler, and by its writer,
// which fills GpArgs.
#pragma once

#include "device.cuh"

namespace psb {

constexpr int kGpThreads = 256;

struct GpArgs {
  GridView g[PSB_MAX_GRIDS];
  double a[PSB_MAX_TERMS], b[PSB_MAX_TERMS], post;        // constant factors
  float a32[PSB_MAX_TERMS], b32[PSB_MAX_TERMS], post32;   // ... rounded to float once
  Dom3 d;
  int color;
  int tx_shift;          // log2 of the threads along x
  int tiles_x, tiles_y;  // blocks along x and y
  unsigned mul_x, mul_y; // b / tiles_x = (b * mul_x) >> shift_x for a block index b
  int shift_x, shift_y;
};

// Indices of the periodic form (i + n) % n: within one period of the grid
// (the launcher checked the domain and the offsets), and in general.
__device__ __forceinline__ int gp_wrap(int i, int n) {
  return i < 0 ? i + n : (i >= n ? i - n : i);
}
__device__ __forceinline__ int gp_mod(int i, int n) { return (i + n) % n; }
__device__ __forceinline__ int gp_clamp(int i, int n) {
  return i < 0 ? 0 : (i > n - 1 ? n - 1 : i);
}

// NC: the grid is not the written one, so its values cannot change while the
// kernel runs.
template <bool NC, typename S>
__device__ __forceinline__ S gp_ld(const S *p) {
  if constexpr (NC) return __ldg(p);
  else return *p;
}

// First point of a thread's U points: U consecutive planes (3-D), rows (2-D)
// or the one point of a 1-D domain. In a coloured pass a thread owns the
// point of its colour in each pair of x columns: the pair starts at x, and
// px is the column's offset in the pair for the first of the U points (it
// alternates from one to the next).
struct GpAt {
  int x, y, z, px;
};

template <int ND, int U, bool COLORED>
__device__ __forceinline__ GpAt gp_position(const GpArgs &q) {
  const unsigned b = blockIdx.x;
  const unsigned row = ND == 1 ? 0 : (unsigned)(((uint64_t)b * q.mul_x) >> q.shift_x);
  const int bx = (int)(b - row * q.tiles_x);
  const int bz = ND < 3 ? 0 : (int)(((uint64_t)row * q.mul_y) >> q.shift_y);
  const int by = (int)row - bz * q.tiles_y;
  const int tx = threadIdx.x & ((1 << q.tx_shift) - 1), ty = threadIdx.x >> q.tx_shift;
  const int xi = (bx << q.tx_shift) + tx, yi = by * (kGpThreads >> q.tx_shift) + ty;
  GpAt at;
  at.x = q.d.lo[0] + (COLORED ? 2 * xi : xi);
  at.y = q.d.lo[1] + (ND == 2 ? yi * U : yi);
  at.z = q.d.lo[2] + bz * (ND == 3 ? U : 1);
  at.px = COLORED ? (q.d.lo[0] + at.y + at.z + q.color) & 1 : 0;
  return at;
}

}  // namespace psb
