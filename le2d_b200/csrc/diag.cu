// FP64 diagnostics of a state: elastic energy, per-field sum of squares and max
// |value|.  The reference has no diagnostics; these define the energy-norm drift
// and the norms reported beside each result.  Every node's contribution is
// formed and summed in double regardless of the storage precision.
#include "le2d_kernels.h"

namespace le2d {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float larger(float m, float x) { return fmaxf(m, fabsf(x)); }
__device__ __forceinline__ double larger(double m, double x) { return fmax(m, fabs(x)); }
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <typename T>
struct Wide;
template <> struct Wide<float> { using type = float4; };
template <> struct Wide<double> { using type = double2; };

// out[0] += sum of energy densities, out[1+k] += sum v_k^2, out[6+k] = max |v_k| (the
// bits of a non-negative double order like the double, so an integer max works).
// Bound by the read of the state: a warp takes 32 vectors of 16 bytes of one row at a time, the
// five fields' loads in flight together; the last vector of a row may reach into its padding,
// whose columns are left out.  The maxima are kept in T (exact).  5 x 4096^2 FP32, one element
// per thread and a 64-bit division each before: 172 us a call, now 75 us (4.5 TB/s).
template <typename T>
__global__ void __launch_bounds__(kThreads) diag_kernel(const T* __restrict__ soa, int nx, int ny,
                                                        long long pitch, long long plane, int chunks,
                                                        double rho, double a_nn, double a_xy,
                                                        double a_s, double* __restrict__ out) {
  using VT = typename Wide<T>::type;
  constexpr int kV = (int)(sizeof(VT) / sizeof(T));
  double acc[11];
  T top[NF];
#pragma unroll
  for (int k = 0; k < 6; ++k) acc[k] = 0.0;
#pragma unroll
  for (int k = 0; k < NF; ++k) top[k] = (T)0;
  const int warps = gridDim.x * (kThreads / 32), items = ny * chunks;  // 32 vectors of a row each
  for (int w = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); w < items; w += warps) {
    const int j = w / chunks;
    const int i = ((w - j * chunks) * 32 + (threadIdx.x & 31)) * kV;
    if (i >= nx) continue;
    const T* s = soa + j * pitch + i;
    VT raw[NF];
#pragma unroll
    for (int k = 0; k < NF; ++k) raw[k] = *reinterpret_cast<const VT*>(s + k * plane);
#pragma unroll
    for (int e = 0; e < kV; ++e) {
      if (i + e >= nx) break;
      double v[NF];
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const T x = reinterpret_cast<const T*>(&raw[k])[e];
        v[k] = (double)x;
        acc[1 + k] += v[k] * v[k];
        top[k] = larger(top[k], x);
      }
      acc[0] += 0.5 * rho * (v[VX] * v[VX] + v[VY] * v[VY]) +
                a_nn * (v[SXX] * v[SXX] + v[SYY] * v[SYY]) + a_xy * v[SXX] * v[SYY] +
                a_s * v[SXY] * v[SXY];
    }
  }
#pragma unroll
  for (int k = 0; k < NF; ++k) acc[6 + k] = (double)top[k];
  __shared__ double red[kThreads / 32][11];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 11; ++k) {
    const double r = k < 6 ? warp_sum(acc[k]) : warp_max(acc[k]);
    if (lane == 0) red[wid][k] = r;
  }
  __syncthreads();
  if (threadIdx.x < 11) {
    const int k = threadIdx.x;
    double r = red[0][k];
    for (int w = 1; w < kThreads / 32; ++w) r = k < 6 ? r + red[w][k] : fmax(r, red[w][k]);
    if (k < 6)
      atomicAdd(out + k, r);
    else
      atomicMax(reinterpret_cast<unsigned long long*>(out + k), (unsigned long long)__double_as_longlong(r));
  }
}

}  // namespace

template <typename T>
cudaError_t launch_diag(const T* soa, int nx, int ny, long long pitch, long long plane,
                        double rho, double a_nn, double a_xy, double a_s, double* out,
                        cudaStream_t s) {
  const int per_warp = 32 * (int)(16 / sizeof(T)), chunks = (nx + per_warp - 1) / per_warp;
  if ((long long)ny * chunks > 0x3fffffffLL) return cudaErrorInvalidValue;
  int blocks = (ny * chunks + kThreads / 32 - 1) / (kThreads / 32);
  if (blocks > 148 * 8) blocks = 148 * 8;
  diag_kernel<T><<<blocks, kThreads, 0, s>>>(soa, nx, ny, pitch, plane, chunks, rho, a_nn, a_xy, a_s, out);
  return cudaGetLastError();
}

template cudaError_t launch_diag<real>(const real*, int, int, long long, long long, double,
                                       double, double, double, double*, cudaStream_t);

}  // namespace le2d
