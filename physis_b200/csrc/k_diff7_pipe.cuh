// 7-point diffusion, several time steps per pass: a register pipeline over z.
//
// A CTA owns an extended tile (the output tile plus an NS-cell halo, NS the
// steps of a pass) and walks a chunk of z. Every thread owns one 16-byte
// vector column of R consecutive rows for the whole walk and keeps, for each
// of the NS stages, the two planes below the newest one in registers, so z
// neighbours never leave the thread: at each turn of the walk stage 1
// computes one plane of the first step from the input, stage 2 one plane of
// the second step from stage 1's last three, and so on, and the last stage
// stores. x neighbours come from the adjacent lanes by warp shuffles, the
// inner y neighbours are the thread's own rows, and only a row group's first
// and last rows go through shared memory, double-buffered, with one CTA
// barrier per turn. Input planes stream through a ring of TMA boxes issued
// S - 2 turns ahead.
//
// What bounds it: instruction issue (66% of the slots at 512^3; the input
// is read and the output written once for NS steps, so DRAM is not the
// limit). Hence the shape: R rows a thread, because the exchange (two loads,
// two stores, two shuffles a row) is paid per thread and row group, not per
// point; rows of 8 to 32 lanes, so that an x extent wastes little of its last
// tile; no branch in the turns between the z faces. Measured, us a step
// against single steps of k_diff7_tma (float, exact / FMA): 512^3 123.4 /
// 102.4 in passes of four (xl 16, 384 threads, 96-plane chunks) against 177;
// 256^3 20.5 / 17.2 against 34 / 33; 128^3 4.7 / 4.2 against 8.5; periodic
// 256^3 in passes of two 28.1 against 40.7; double 256^3 30.9 / 28.8 in
// passes of two against 48.
//
// The outermost NS cells of the extended tile become invalid one per stage
// and are not stored; at a clamped face the face rule stands in for the halo,
// so the tile starts at the face itself. Every point of every stage is
// computed with the single-step arithmetic and face rules: the results are
// those of NS single steps, bit for bit.
#pragma once

#include "k_diffusion7.cuh"

namespace psb {

struct PipeGeom {
  int ax0, ay0, az0;       // tensor-map coordinates of logical (0, 0, 0)
  int xl_shift;            // log2 of the lanes (16-byte vectors) of a row
  int rows;                // rows of the extended tile
  int bx, nbox;            // TMA boxes of a plane: nbox of bx x rows elements
  int ex0, ey0, sx, sy;    // start of the first extended tile, stride of tiles
  int tiles_x, tiles_y, zchunk;
  int stages, plane_bytes;
};

// Points at each x end of an extended tile that it does not store: the NS
// that become invalid, rounded up where tile starts, NS apart from a multiple
// of the vector, would leave 16 bytes.
__host__ __device__ constexpr int pipe_hx(int ns, int v) {
  return 2 * ns % v == 0 ? ns : (ns + v - 1) / v * v;
}

template <int I>
struct PipeIdx {
  static constexpr int value = I;
};

template <typename T, int NS, int R, bool GHOST, bool PERIODIC, bool FAST>
__device__ __forceinline__ void diff7_pipe(const CUtensorMap *tin, const GridView out, int nx,
                                           int ny, int nz, const C7<T> k7, const PipeGeom geo,
                                           int *err, unsigned char *smem) {
  constexpr int V = Vec16<T>::N;
  constexpr int HX = pipe_hx(NS, V);
  const int S = geo.stages;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);
  unsigned char *ring = smem + 128;
  const int nthr = blockDim.x, tid = threadIdx.x;
  const int XL = 1 << geo.xl_shift;
  const int lx = tid & (XL - 1), rg = tid >> geo.xl_shift;
  // Published first and last rows of stages 1 .. NS-1 ([stage][parity][first,
  // last][thread]).
  Vec16<T> *edges = reinterpret_cast<Vec16<T> *>(ring + (size_t)S * geo.plane_bytes);

  int b = blockIdx.x;
  const int tile_x = b % geo.tiles_x;
  b /= geo.tiles_x;
  const int tile_y = b % geo.tiles_y;
  const int zb = (b / geo.tiles_y) * geo.zchunk;
  const int nzl = min(zb + geo.zchunk, nz) - zb;
  const int nit = nzl + 2 * NS;  // input planes zb - NS .. zb + nzl + NS - 1
  const int W = XL * V;
  const int xe = geo.ex0 + tile_x * geo.sx;
  // Clamped: the last tile ends at the face, so that the face row is the
  // last row of its group (see the face rules below).
  const int yt = geo.ey0 + tile_y * geo.sy;
  const int ye = PERIODIC ? yt : min(yt, max(0, ny - geo.rows));
  const int xg0 = xe + lx * V, yg0 = ye + rg * R;
  // The points this tile stores.
  int xlo, xhi, ylo, yhi;
  if (PERIODIC) {
    xlo = max(0, xe + HX);
    xhi = min(nx, xe + W - HX);
    ylo = max(0, yt + NS);
    yhi = min(ny, yt + geo.rows - NS);
  } else {
    xlo = xe == 0 ? 0 : xe + HX;
    xhi = xe + W >= nx ? nx : xe + W - HX;
    ylo = yt == 0 ? 0 : yt + NS;
    yhi = yt + geo.rows >= ny ? ny : yt + geo.rows - NS;
  }
  const bool xall = xg0 >= xlo && xg0 + V <= xhi;
  const bool xany = xg0 + V > xlo && xg0 < xhi;
  bool row_in[R];
#pragma unroll
  for (int r = 0; r < R; r++) row_in[r] = xany && yg0 + r >= ylo && yg0 + r < yhi;
  // Clamped faces. A neighbour outside the grid is the point itself: w of
  // x = 0 and e of a vector that ends at x = nx-1 are selects; a row whose
  // last point is inside a vector (xr), and a column whose last row is inside
  // a thread's rows (yr), continue one point past the face with the face
  // value, copied there when a plane is produced; the first and last rows of
  // the grid otherwise read their own row in place of the neighbour group's.
  // GHOST: a grid that needs the copies (the others leave them out).
  const bool face_w = !PERIODIC && xg0 == 0, face_e = !PERIODIC && xg0 + V == nx;
  const bool xr = !PERIODIC && nx % V != 0 && xe + W > nx;
  const int xghost = nx - xg0;  // element at x = nx
  const int yghost = ny - yg0;  // row at y = ny
  const bool yr = !PERIODIC && yghost > 0 && yghost < R;
  auto ghosts = [&](Vec16<T>(&q)[R]) {
    if (xr) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int v = 1; v < V; v++)
          if (v == xghost) q[r].v[v] = q[r].v[v - 1];
    }
    if (yr) {
#pragma unroll
      for (int r = 1; r < R; r++)
        if (r == yghost) q[r] = q[r - 1];
    }
  };
  const K7<T> kk = make_k7(k7);
  const uint32_t bytes = (uint32_t)geo.plane_bytes;
  const int box_bytes = geo.bx * geo.rows * (int)sizeof(T);
  auto issue = [&](int j, int slot) {  // input plane j of the walk (one thread)
    int z = zb - NS + j;
    if (PERIODIC) z = z < 0 ? z + nz : (z >= nz ? z - nz : z);  // the wrapped plane itself
    mbar_arrive_expect_tx(&full[slot], bytes);
    for (int i = 0; i < geo.nbox; i++)
      tma_load_3d(ring + (size_t)slot * geo.plane_bytes + (size_t)i * box_bytes, tin, &full[slot],
                  xe + geo.ax0 + i * geo.bx, ye + geo.ay0, z + geo.az0);
  };
  if (tid == 0) {
    for (int i = 0; i < S; i++) mbar_init(&full[i], 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (tid == 0) {
    tma_prefetch_desc(tin);
    for (int j = 0; j < S && j < nit; j++) issue(j, j);
  }

  // Offsets of this thread's vector in a plane: column block, then rows.
  const int col = lx * V;
  const int pcol = (col / geo.bx) * (geo.bx * geo.rows) + col % geo.bx;
  const int prow = rg * R;
  const int off_own = pcol + prow * geo.bx;
  const int off_n = pcol + max(prow - 1, 0) * geo.bx;
  const bool face_s = !PERIODIC && yghost == R;  // the last row is y = ny-1
  const int off_s = pcol + (face_s ? prow + R - 1 : min(prow + R, geo.rows - 1)) * geo.bx;
  // Published row above this group (the group above's last row; the grid's
  // first row is its own neighbour) and below it.
  const int e_n = rg > 0 ? nthr + tid - XL : tid;
  const int e_s = face_s || tid + XL >= nthr ? nthr + tid : tid + XL;

  Vec16<T> P[NS][3][R];  // planes of stages 0 .. NS-1, by turn modulo 3
#pragma unroll
  for (int s = 0; s < NS; s++)
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int v = 0; v < V; v++) P[s][i][r].v[v] = (T)0;
  bool bad = false;
  int slot = 0, prev = 0;  // ring slots of this and the previous plane
  uint32_t round = 0;
  T *dst0 = (T *)out.origin + xg0 + (int64_t)yg0 * out.sy + (int64_t)(zb - 2 * NS) * out.sz;

  // Turn k of the walk; km = k modulo 3. EDGE: turns before the last stage
  // has its three planes, or in which a stage meets a clamped z face. The
  // walk between them has no such branches, which would split its schedule
  // (512^3 float exact: 159 us a step with them, 126 us without).
  auto turn = [&](int k, auto km_, auto edge_) __attribute__((always_inline)) {
    constexpr int A = decltype(km_)::value, C = (A + 2) % 3, B = (A + 1) % 3;
    constexpr bool EDGE = decltype(edge_)::value != 0;
    if (!bad && !mbar_wait_bounded(&full[slot], round & 1)) {
      bad = true;  // carry on without waiting: the walk is bounded
      atomicExch(err, 1);
    }
    const T *pk = reinterpret_cast<const T *>(ring + (size_t)slot * geo.plane_bytes);
    const T *pp = reinterpret_cast<const T *>(ring + (size_t)prev * geo.plane_bytes);
#pragma unroll
    for (int r = 0; r < R; r++) P[0][A][r] = lds16(pk + off_own + r * geo.bx);
    if constexpr (GHOST) ghosts(P[0][A]);
    const int par = k & 1;
#pragma unroll
    for (int s = 1; s <= NS; s++) {
      // The planes below, at and above the one this stage computes.
      Vec16<T>(&pb)[R] = P[s - 1][B];
      Vec16<T>(&pc)[R] = P[s - 1][C];
      Vec16<T>(&pt)[R] = P[s - 1][A];
      // Publish what the neighbours need of the next turn's centre plane.
      if (s > 1) {
        Vec16<T> *e = edges + (size_t)(((s - 2) * 2 + par) * 2) * nthr + tid;
        stg16(reinterpret_cast<T *>(e), pt[0]);
        stg16(reinterpret_cast<T *>(e + nthr), pt[R - 1]);
      }
      if (EDGE && k < 2 * s) continue;  // uniform: this stage has no three planes yet
      const int z = zb - NS + k - s;
      Vec16<T> vn, vs;
      if (s == 1) {
        vn = lds16(pp + off_n);
        vs = lds16(pp + off_s);
      } else {
        const Vec16<T> *e = edges + (size_t)(((s - 2) * 2 + (par ^ 1)) * 2) * nthr;
        vn = lds16(reinterpret_cast<const T *>(e + e_n));
        vs = lds16(reinterpret_cast<const T *>(e + e_s));
      }
      T wl[R], er[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        wl[r] = __shfl_up_sync(0xffffffffu, pc[r].v[V - 1], 1);
        er[r] = __shfl_down_sync(0xffffffffu, pc[r].v[0], 1);
      }
      if (!PERIODIC) {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (face_w) wl[r] = pc[r].v[0];
          if (face_e) er[r] = pc[r].v[V - 1];
        }
        if (EDGE && z == 0) {
#pragma unroll
          for (int r = 0; r < R; r++) pb[r] = pc[r];
        }
        if (EDGE && z == nz - 1) {
#pragma unroll
          for (int r = 0; r < R; r++) pt[r] = pc[r];
        }
      }
      Vec16<T> res[R];
#pragma unroll
      for (int r = 0; r < R; r++)
        res[r] = diff7_row<T, FAST>(kk, pc[r], wl[r], er[r], r == 0 ? vn : pc[r - 1],
                                    r == R - 1 ? vs : pc[r + 1], pb[r], pt[r], 0u);
      if (s < NS) {
#pragma unroll
        for (int r = 0; r < R; r++) P[s < NS ? s : 0][A][r] = res[r];
        if constexpr (GHOST) ghosts(P[s < NS ? s : 0][A]);
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (!row_in[r]) continue;
          T *dst = dst0 + r * out.sy;
          if (xall) {
            stg16(dst, res[r]);
          } else {
#pragma unroll
            for (int e = 0; e < V; e++)
              if (xg0 + e >= xlo && xg0 + e < xhi) dst[e] = res[r].v[e];
          }
        }
      }
    }
    dst0 += out.sz;
    __syncthreads();  // edges visible; the previous plane's slot is free
    if (tid == 0 && k >= 1 && k - 1 + S < nit) issue(k - 1 + S, prev);
    prev = slot;
    if (++slot == S) {
      slot = 0;
      round++;
    }
  };
  const PipeIdx<0> I0;
  const PipeIdx<1> I1;
  const PipeIdx<2> I2;
  for (int k = 0; k < nit; k += 3) {
    // The planes these three turns compute lie in z0 .. z1.
    const int z0 = zb - 2 * NS + k, z1 = zb - NS + k + 1;
    if (k >= 2 * NS && k + 3 <= nit && (PERIODIC || (z0 > 0 && z1 < nz - 1))) {
      turn(k, I0, I0);
      turn(k + 1, I1, I0);
      turn(k + 2, I2, I0);
    } else {
      turn(k, I0, I1);
      if (k + 1 < nit) turn(k + 1, I1, I1);
      if (k + 2 < nit) turn(k + 2, I2, I1);
    }
  }
  if constexpr (PERIODIC) {
    // The output's halo for the next pass: the points within two of an x or y
    // face go to their images too, corners included (planes beyond a z face
    // are loaded from where they wrap to). Copied from the CTA's own stores
    // after the walk: image code inside the turns outgrew the instruction
    // cache (256^3 float: 37 us a step).
    __syncthreads();
    T *o = (T *)out.origin;
    const int nrows = yhi - ylo, ncols = xhi - xlo;
    constexpr int U = 8;  // independent copies in flight per thread
    // x faces: columns 0 and 1 (side 0), nx-2 and nx-1 (side 1).
    for (int side = 0; side < 2 && nrows > 0; side++) {
      const int xs = side ? nx - 2 : 0, xt = side ? -nx : nx;
      if (xs + 1 < xlo || xs >= xhi) continue;
      const int total = nrows * nzl * 2;
      for (int i0 = tid; i0 < total; i0 += U * nthr) {
        T v[U], *p[U];
        int y[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * nthr, x = xs + (i & 1), q = i >> 1;
          y[u] = ylo + q % nrows;
          in[u] = i < total && x >= xlo && x < xhi;
          p[u] = o + x + (int64_t)y[u] * out.sy + (int64_t)(zb + q / nrows) * out.sz;
          if (in[u]) v[u] = __ldcg(p[u]);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (!in[u]) continue;
          p[u][xt] = v[u];
          if (y[u] < 2) p[u][xt + ny * out.sy] = v[u];
          if (y[u] >= ny - 2) p[u][xt - ny * out.sy] = v[u];
        }
      }
    }
    // y faces: rows 0 and 1, ny-2 and ny-1.
    for (int side = 0; side < 2 && ncols > 0; side++) {
      const int ys = side ? ny - 2 : 0;
      const int64_t to = (side ? -ny : ny) * out.sy;
      if (ys + 1 < ylo || ys >= yhi) continue;
      const int total = ncols * nzl * 2;
      for (int i0 = tid; i0 < total; i0 += U * nthr) {
        T v[U], *p[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * nthr, q = i / ncols, y = ys + (q & 1);
          in[u] = i < total && y >= ylo && y < yhi;
          p[u] = o + xlo + i % ncols + (int64_t)y * out.sy + (int64_t)(zb + (q >> 1)) * out.sz;
          if (in[u]) v[u] = __ldcg(p[u]);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (in[u]) p[u][to] = v[u];
      }
    }
  }
  if (bad && tid == 0)  // copies that were not waited for: let them land (bounded)
    for (int i = 0; i < S && i < nit; i++) {
      const int last = (nit - 1 - i) / S;
      const long long t0 = clock64();
      while (!mbar_try_wait(&full[i], last & 1) && clock64() - t0 < 200000000LL) {
      }
    }
}

}  // namespace psb
