// Small grids: several time steps per launch on block tiles (tile.cuh).
//
// What bounds it.  A launch costs A + B x steps per wave of tiles: A (launch, tile and halo
// read from L2, instruction fetch, write) is 2.1 to 5.8 us, and a step's B follows the nodes
// of a tile.  More steps per launch share A but widen the halo that neighbouring tiles compute
// twice, so the best tile and depth depend on the grid, and plan_tiles() takes them from a
// table of measured A and B.  Measured (us a step, this path / the strip march as it was
// planned before, 32-row segments): FP32 100 x 67 1.2 / 18.2, 256^2 1.6 / 18.4, 512^2 3.3 /
// 18.5, 700 x 600 4.5 / 18.5, 1200 x 900 11.6 / 20.3; FP64 100 x 67 2.6 / 24.0, 256^2 4.1 /
// 24.4, 512^2 9.4 / 24.6, 700 x 600 16.1 / 24.6.
//
// Launches are programmatic: a launch's blocks may come up while the one before drains and
// wait for it (griddepcontrol) only before they read, with their addresses, masks and row table
// formed: waiting at the kernel's start cost 0.4 to 0.9 us a launch (100 x 67 1.41 / 1.23, 512^2
// 3.48 / 3.34 us a step).  Without programmatic launches every launch of a stream took whole
// multiples of about 2 us (100 x 67 1.4 against 2.1 us a step, 512^2 3.9 against 4.3); a captured
// graph did about as well but has to be captured first.
#include <atomic>
#include <cmath>
#include <type_traits>

#include "tile.cuh"

namespace le2d {

namespace {

template <typename T>
struct TileParams {
  march::GridRef<T> g;
  int ntx, nty, out_x;  // tiles across and down, columns a tile writes
  int depth, steps;
  StepConsts<T> c;
  YPairs yq;
};

__device__ __forceinline__ const YPairs& ycons(const TileParams<float>& p) { return p.yq; }
__device__ __forceinline__ const Sweep<double>& ycons(const TileParams<double>& p) { return p.c.y; }

template <typename T, int V, int R, int W>
__global__ void __launch_bounds__(W * 32, 1) block_tile_kernel(const __grid_constant__ TileParams<T> p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cudaTriggerProgrammaticLaunchCompletion();
  const int tx = blockIdx.x % p.ntx, ty = blockIdx.x / p.ntx;
  const int ox0 = tx * p.out_x, ox1 = min(ox0 + p.out_x, p.g.nx);
  // rows shared out evenly (le_step_soa's far end needs at least 3 in the last tile)
  const int oy0 = (int)((long long)ty * p.g.ny / p.nty), oy1 = (int)((long long)(ty + 1) * p.g.ny / p.nty);
  // loads past L1: under a programmatic launch the data may be older there
  march::block_tile<T, V, R, W, true, false, true>(p.g, p.c.x, ycons(p), ox0, ox1, oy0, oy1, p.depth, p.steps,
                                                   reinterpret_cast<T*>(smem_raw),
                                                   march::BlockTap<T>{nullptr, -1, 1, 1});
}

// Tile shapes: V columns per lane, R rows per warp, W warps; A and B of the launch time above
// (us), fitted to launches of one wave with 1 to 6 steps.  Small tiles for the smallest grids,
// whose launches they end soonest; large ones where the halo's share counts.  Register bounds
// without (FP32) or with few spills: 128 registers at 16 warps, 168 at 12.  Other shapes timed
// and not kept (same grids): 4 columns per lane (372 bytes of spills), 64 x 32 tiles two to an
// SM (FP32 1200 x 900 11.6 against 11.9 us, slower on the others), FP64 64 x 48 on 16 warps
// (512^2 10.2 against 9.6), FP64 one column per lane (512^2 11.5).
struct TileShape {
  int V, R, W;
  double a, b;
};
template <typename T>
struct Shapes;
template <>
struct Shapes<float> {
  static constexpr TileShape s[] = {{2, 4, 16, 4.0, 2.62}, {2, 4, 12, 3.6, 1.68}, {2, 2, 16, 3.3, 0.98}, {2, 2, 8, 2.1, 0.62}};
};
template <>
struct Shapes<double> {
  static constexpr TileShape s[] = {{2, 4, 12, 5.8, 6.36}, {2, 2, 12, 3.1, 3.13}, {2, 1, 16, 2.5, 2.05}};
};
constexpr int kMaxDepth = 6;

template <typename T>
constexpr int shape_count() { return (int)(sizeof(Shapes<T>::s) / sizeof(TileShape)); }

template <typename T, int S>
struct TileKernel {
  static constexpr TileShape c = Shapes<T>::s[S];
  // at least 116 KB: one block to an SM (two would crowd some SMs and leave others idle)
  static constexpr size_t smem() {
    constexpr size_t need = march::block_tile_smem<T, c.V, c.R, c.W>();
    return need > (116u << 10) ? need : (116u << 10);
  }
  static cudaError_t launch(const TileParams<T>& p, int blocks, cudaStream_t s) {
    auto* fn = block_tile_kernel<T, c.V, c.R, c.W>;
    // shared memory above 48 KB is opted into once per device (devices 0..63)
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !(done.load() >> dev & 1)) {
      const cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem());
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) done.fetch_or(1ull << dev);
    }
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(blocks);
    lc.blockDim = dim3(c.W * 32);
    lc.dynamicSmemBytes = smem();
    lc.stream = s;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, fn, p);
  }
};

template <typename T, int S = 0>
cudaError_t launch_shape(int shape, const TileParams<T>& p, int blocks, cudaStream_t s) {
  if constexpr (S < shape_count<T>()) {
    if (shape == S) return TileKernel<T, S>::launch(p, blocks, s);
    return launch_shape<T, S + 1>(shape, p, blocks, s);
  } else {
    return cudaErrorInvalidValue;
  }
}

}  // namespace

// The tile shape and depth with the least modelled time per step, if that is below the strip
// march's.  A launch of n tiles on `sms` SMs takes its waves' time, each wave after the first
// at 0.92 of it (blocks start as others end).  The model's choice was within 3 % of the
// fastest of all shapes and depths measured on each of the grids named above and 900^2.
// The strip march's time per step is fitted on 700 x 600 to 2048^2 (its best segments, whole or
// in halves): FP32 7.0 + 5.45 us per million nodes (900^2 12.2, 1200 x 900 12.7, 2048^2 29.9
// us), FP64 11 + 17.8 us (700 x 600 19.3, 1200 x 900 30.4, 2048^2 85 us).  So FP32 grids cross over
// at about 1.2 million nodes (1200 x 900 11.6 on tiles, 12.7 on strips; 1500^2 23 and 20.7), FP64
// ones at 0.6 million (700 x 600 16.1 and 19.3; 900^2 27.5 and 25.0).
template <typename T>
TilePlan plan_tiles(int nx, int ny, int sms) {
  TilePlan best;
  const double mnodes = (double)nx * ny * 1e-6;
  double least = sizeof(T) == 4 ? 7.0 + 5.45 * mnodes : 11.0 + 17.8 * mnodes;
  for (int k = 0; k < shape_count<T>(); ++k) {
    const TileShape& c = Shapes<T>::s[k];
    for (int d = 1; d <= kMaxDepth; ++d) {
      const int out_x = 32 * c.V - 4 * d, out_y = c.R * c.W - 4 * d;
      if (out_x < 4 || out_y < 4) break;
      const long long ntx = (nx + out_x - 1) / out_x, nty = (ny + out_y - 1) / out_y;
      const double waves = std::ceil((double)ntx * nty / sms);
      const double t = (c.a + c.b * d) * (1.0 + 0.92 * (waves - 1.0)) / d;
      if (t < least) {
        least = t;
        best.shape = k;
        best.depth = d;
        best.out_x = out_x;
        best.rows = c.R * c.W;
        best.cols = 32 * c.V;
        best.ntx = (int)ntx;
        best.nty = (int)nty;
      }
    }
  }
  return best;
}

template <typename T>
cudaError_t launch_tiles(const T* src, T* dst, int nx, int ny, long long pitch, long long plane,
                         const StepConsts<T>& c, int far_rot, const TilePlan& plan, int steps, cudaStream_t s) {
  if (steps < 1 || steps > plan.depth) return cudaErrorInvalidValue;
  TileParams<T> p;
  p.g = march::GridRef<T>{src, dst, nx, ny, pitch, plane, far_rot};
  p.ntx = plan.ntx;
  p.nty = plan.nty;
  p.out_x = plan.out_x;
  p.depth = plan.depth;
  p.steps = steps;
  p.c = c;
  p.yq = YPairs{};
  if constexpr (std::is_same<T, float>::value) p.yq = make_ypairs(c.y);
  return launch_shape<T>(plan.shape, p, plan.ntx * plan.nty, s);
}

#ifdef LE2D_CHECK
unsigned long long check_violations_tiles() {
  unsigned long long v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, march::g_check_violations, sizeof(v)) != cudaSuccess ||
      cudaMemcpyToSymbol(march::g_check_violations, &zero, sizeof(zero)) != cudaSuccess) {
    cudaGetLastError();
    return ~0ULL;  // unreadable: reported as violations
  }
  return v;
}
#endif

#define LE2D_INST(T)                                                                              \
  template TilePlan plan_tiles<T>(int, int, int);                                                 \
  template cudaError_t launch_tiles<T>(const T*, T*, int, int, long long, long long,              \
                                       const StepConsts<T>&, int, const TilePlan&, int, cudaStream_t);
LE2D_INST(real)
#undef LE2D_INST

}  // namespace le2d
