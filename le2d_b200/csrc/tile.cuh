// Block tiles: several time steps of a small grid per launch.  A block holds a tile of the
// grid -- W warps stacked in y, each with R rows of 32 * V columns, V per lane -- in registers
// for the whole launch and advances it step by step; the tile shrinks by the stencil's reach
// (two nodes each way) with every step, so a launch of S steps reads 2 S halo nodes around
// the nodes it writes.
//
// Per step a warp x-sweeps its rows in registers (neighbour columns by shuffles, as in
// march.cuh), puts the fields that the y-sweep reads across rows (vy, syy, vx, sxy) into
// shared memory, and after one block barrier y-sweeps its R rows: the rows from two above its
// first to two below its last go through the y-pipeline (YPipe, fully unrolled, so that what
// only the rows outside need is never computed).  The exchange is double-buffered: a warp can
// write the next step's rows while others still read this one's.
//
// Why not the strip march here: a strip's rows are one serial chain, about 0.9 us a row at low
// occupancy, so a launch cannot end sooner than its segment's rows plus ten allow, and a
// small grid has too few strips to hide that.
//
// Ends of the grid.  In y the exchange is read at clamped rows (past the last row, rows m - 5
// for le_step_soa's far end), as the strip march reads its source rows.  In x the faces at or
// beyond the ends are masked (FP32) or their invariants and fluxes replaced by the edge
// column's (FP64), see sweep_x_lane_packed / sweep_x_lane_exact.  Rows and columns that are
// neither in the grid nor valid any more hold finite values that nothing valid reads.
// Results are bitwise those of the strip march.
#pragma once

#include "march.cuh"

namespace le2d {
namespace march {

constexpr int kXchg = 4;  // exchanged fields: vy, syy, vx, sxy

template <typename T, int V, int R, int W>
__host__ __device__ constexpr size_t block_tile_smem() {
  return (size_t)2 * R * W * kXchg * 32 * V * sizeof(T);
}

// The rows of the exchange a warp's y-sweep reads, one byte each: rows j0 - 2 .. j0 + R + 1 of
// the grid, clamped to it and to the tile (a clamp a row and step would be 6 instructions each,
// 4 % of a step).
template <int R>
struct BlockRows {
  static constexpr int kWords = (R + 4 + 3) / 4;
  unsigned w[kWords];
  __device__ __forceinline__ void set(int j0, int y_tile, int rows, int ny, int far_rot) {
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = 0;
#pragma unroll
    for (int i = 0; i < R + 4; ++i) {
      const int j = min(max(source_row(j0 - 2 + i, ny, far_rot) - y_tile, 0), rows - 1);
      w[i / 4] |= (unsigned)j << (8 * (i % 4));
    }
  }
  __device__ __forceinline__ unsigned operator[](int i) const { return __byte_perm(w[i / 4], 0, 0x4440 + i % 4); }
};

// The y-sweep of a warp's rows f (x-swept); `buf` the exchange of this step (lane's first
// column).
template <typename T, int V, int R, typename CY>
__device__ __forceinline__ void block_sweep_y(T (&f)[R][NF][V], const T* buf, const BlockRows<R>& rows, const CY& cy) {
  using VT = typename Vec<T, V>::type;
  constexpr int kIn = 32 * V;
  YPipe<T, V> yp;
  yp.init();
  T cur[NF][V], pvy[V], psyy[V], pvx[V], psxy[V];
#pragma unroll
  for (int m = -2; m < R + 2; ++m) {
    const T* p = buf + rows[m + 2] * (kXchg * kIn);
    unpack(*reinterpret_cast<const VT*>(p), cur[VY]);
    unpack(*reinterpret_cast<const VT*>(p + kIn), cur[SYY]);
    unpack(*reinterpret_cast<const VT*>(p + 2 * kIn), cur[VX]);
    unpack(*reinterpret_cast<const VT*>(p + 3 * kIn), cur[SXY]);
    if (m > -2) {
      yp.left(cur, pvy, psyy, pvx, psxy, cy);
      if (m >= 2) yp.apply(f[m - 2], cy);
      yp.right(cy);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      pvy[v] = cur[VY][v];
      psyy[v] = cur[SYY][v];
      pvx[v] = cur[VX][v];
      psxy[v] = cur[SXY][v];
    }
  }
}

// A receiver line of a batched instance: vx and vy of `row` after every `every` steps, the next
// sample `until` (1 .. every) steps ahead, at out[0 .. pitch) and out[pitch .. 2 pitch); the
// samples follow each other.
template <typename T>
struct BlockTap {
  T* out;
  int row, every, until;
};

// Advances the tile that writes columns [ox0, ox1), rows [oy0, oy1) by `steps` steps; its
// first column and row lie 2 * depth before ox0 and oy0 (depth >= steps; ox0 a multiple of V).
// ox1 - ox0 + 4 depth <= 32 V and oy1 - oy0 + 4 depth <= R W.  TAP: records the tile's part of a
// receiver line.  WAIT: waits for the launch before, after what does not depend on it.  Called by
// the whole block.
template <typename T, int V, int R, int W, bool COHERENT, bool TAP, bool WAIT, typename CY>
__device__ __forceinline__ void block_tile(const GridRef<T>& g, const Sweep<T>& cx, const CY& cy, int ox0,
                                           int ox1, int oy0, int oy1, int depth, int steps, T* smem,
                                           BlockTap<T> tap) {
  using VT = typename Vec<T, V>::type;
  constexpr int kIn = 32 * V;
  constexpr int kBuf = R * W * kXchg * kIn;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int y_tile = oy0 - 2 * depth;
  const int j0 = y_tile + warp * R;
  const int col0 = ox0 - 2 * depth + lane * V;
  const bool col_in = col0 >= 0 && col0 < g.nx;

  float em[V + 1];  // FP32: face e lies between columns col0 + e - 1 and col0 + e
#pragma unroll
  for (int e = 0; e <= V; ++e) em[e] = col0 + e >= 1 && col0 + e < g.nx ? 1.0f : 0.0f;
  BlockRows<R> rows;
  rows.set(j0, y_tile, R * W, g.ny, g.far_rot);
  if constexpr (WAIT) cudaGridDependencySynchronize();  // the launch before wrote the state read here

  T f[R][NF][V];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int j = j0 + i;
    const bool in = col_in && j >= 0 && j < min(g.ny, oy1 + 2 * depth);
    const T* row = g.src + (long long)j * g.pitch + col0;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      VT v{};
      if (in && in_src(g, row + k * g.plane, V))
        v = load_state<COHERENT>(reinterpret_cast<const VT*>(row + k * g.plane));
      unpack(v, f[i][k]);
#pragma unroll
      for (int e = 1; e < V; ++e) f[i][k][e] = col0 + e < g.nx ? f[i][k][e] : (T)0;
    }
  }

  T* buf = smem;
  for (int s = 0; s < steps; ++s) {
    // rows the remaining steps need of this one, and of its x-sweep
    const int rem = 2 * (steps - 1 - s);
    const int ylo = max(oy0 - rem, 0), yhi = min(oy1 + rem, g.ny);
    T* mine = buf + warp * R * (kXchg * kIn) + lane * V;
    if (j0 < yhi + 2 && j0 + R > ylo - 2 && j0 < g.ny && j0 + R > 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if constexpr (sizeof(T) == 8)
          sweep_x_lane_exact<V, true>(f[i], cx, col0, g.nx);
        else
          sweep_x_lane_packed<V, true>(f[i], cx, em);
        T* p = mine + i * (kXchg * kIn);
        *reinterpret_cast<VT*>(p) = pack(f[i][VY]);
        *reinterpret_cast<VT*>(p + kIn) = pack(f[i][SYY]);
        *reinterpret_cast<VT*>(p + 2 * kIn) = pack(f[i][VX]);
        *reinterpret_cast<VT*>(p + 3 * kIn) = pack(f[i][SXY]);
      }
    }
    __syncthreads();
    if (j0 < yhi && j0 + R > ylo)
      block_sweep_y<T, V, R>(f, buf + lane * V, rows, cy);
    buf = buf == smem ? smem + kBuf : smem;
    if (TAP && tap.out != nullptr && --tap.until == 0) {
      tap.until = tap.every;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (j0 + i == tap.row && tap.row >= oy0 && tap.row < oy1 && col0 >= ox0 && col0 < ox1 &&
            in_line(col0, V, g.pitch)) {
          *reinterpret_cast<VT*>(tap.out + col0) = pack(f[i][VX]);
          *reinterpret_cast<VT*>(tap.out + g.pitch + col0) = pack(f[i][VY]);
        }
      }
      tap.out += 2 * g.pitch;
    }
  }

#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int j = j0 + i;
    const bool in = j >= oy0 && j < oy1 && col0 >= ox0 && col0 < ox1;
    T* row = g.dst + (long long)j * g.pitch + col0;
#pragma unroll
    for (int k = 0; k < NF; ++k)
      store_if(in && in_dst(g, row + k * g.plane, V), reinterpret_cast<VT*>(row + k * g.plane), pack(f[i][k]));
  }
}

}  // namespace march
}  // namespace le2d
