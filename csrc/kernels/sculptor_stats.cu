// Sculptor calibration statistics on the device.
//  * layer_sumsq: sum of squares of every recorded layer in one launch (-> L2 norms for the Welford
//    norm statistics and the kNN pair schedule);
//  * pair_update: for every scheduled pair of equal-size layers, one Welford step of the element-wise
//    means, second moments and co-moment (five FP32 state vectors per pair, resident on the device);
//  * pair_finalize: reduces a pair's state to the scalars the mask builder needs — the element-
//    averaged Pearson correlation and the element-averaged regression (alpha, beta) in both
//    directions — with FP64 accumulation.
// All pairs of a step are processed by ONE launch each (grid.y = pair).
//
// Replaces the host loops of nangila-core/src/sculptor.rs: record (:238-255, sum of squares),
// StreamingCorrelation::update (:108-141), correlation (:144-170) and coupling (:428-474), keeping
// their validity thresholds (1e-10 on sqrt(var_i var_j) and on var_driver).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "nangila_kernels.h"
#include "quant.cuh"

namespace nangila {
namespace {

constexpr int kThreads = 256;

// Where a launch takes its descriptors from: a device array of the caller's, or the kernel's own parameters (a step's
// descriptors are new every time, and a copy of a few hundred bytes to the device costs the host more than the launch).
template <typename Desc>
struct FromMemory {
  static constexpr bool kGridMayBeShort = true;
  const Desc* d;
};
template <typename Desc>
struct FromParams {
  static constexpr bool kGridMayBeShort = false;
  static constexpr int kMax = 64;
  Desc d[kMax];
};

__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < kThreads / 32; ++i) r += sh[i];
  __syncthreads();
  return r;  // valid in thread 0
}

// Sum of squares in FP64. Bound by HBM (2 or 4 bytes an element) and, for layers of a megabyte, by latency: a thread takes
// eight neighbouring elements per step with one or two 16-byte loads, two steps in flight.
constexpr int kSumStep = kThreads * 8;
template <typename T>
__device__ __forceinline__ double sumsq(const T* p, int64_t n) {
  double acc = 0.0;
  const bool vec = (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
#pragma unroll 2
  for (int64_t i = int64_t(blockIdx.x) * kSumStep + threadIdx.x * 8; i < n; i += int64_t(gridDim.x) * kSumStep) {
    float v[8];
    if (vec) {
      dev::load8_guarded<T>(p, i, n, v);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = i + k < n ? dev::Vec16<T>::to_float(p[i + k]) : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += double(v[k]) * double(v[k]);
  }
  return acc;
}
template <typename Source>
__global__ void __launch_bounds__(kThreads) layer_sumsq_kernel(const __grid_constant__ Source layers, double* out) {
  __shared__ double sh[kThreads / 32];
  const NangilaLayerDesc L = layers.d[blockIdx.y];
  const double acc = L.dtype == NANGILA_F32    ? sumsq(static_cast<const float*>(L.data), L.numel)
                     : L.dtype == NANGILA_BF16 ? sumsq(static_cast<const __nv_bfloat16*>(L.data), L.numel)
                                               : sumsq(static_cast<const __half*>(L.data), L.numel);
  const double s = block_sum(acc, sh);
  if (threadIdx.x == 0 && s != 0.0) atomicAdd(&out[blockIdx.y], s);
}

// state layout per pair: mean_i[n], mean_j[n], m2_i[n], m2_j[n], co[n]
//
// Bound by HBM: 40 bytes of state an element, in and out, and the two gradients. A CTA takes one tile of 1024 elements and ends (the grid
// covers the largest pair): four elements a thread, one CTA width apart, so that loads and stores are whole lines whatever the
// alignment of the five vectors (numel may be odd), and all of them are issued before the first is used: with one element in
// flight the 28 pairs of eight 589 824-element bf16 layers took 210 us, 3.2 TB/s; now 110 us, 6.1 TB/s.
constexpr int kPer = 4;
constexpr int kPairTile = kThreads * kPer;
template <typename T>
__device__ __forceinline__ void pair_tile(const NangilaPairDesc& P, int64_t first) {
  const int64_t n = P.numel;
  const T* xi = static_cast<const T*>(P.data_i);
  const T* xj = static_cast<const T*>(P.data_j);
  const float inv_n = 1.0f / float(P.count_after);
  float vi[kPer], vj[kPer], st[5][kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int64_t k = first + u * kThreads;
    if (k < n) {
      vi[u] = dev::Vec16<T>::to_float(xi[k]);
      vj[u] = dev::Vec16<T>::to_float(xj[k]);
#pragma unroll
      for (int q = 0; q < 5; ++q) st[q][u] = P.state[q * n + k];
    }
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int64_t k = first + u * kThreads;
    if (k < n) {
      const float di = vi[u] - st[0][u], dj = vj[u] - st[1][u];
      const float mi = __fmaf_rn(di, inv_n, st[0][u]), mj = __fmaf_rn(dj, inv_n, st[1][u]);
      P.state[k] = mi;
      P.state[n + k] = mj;
      P.state[2 * n + k] = __fmaf_rn(di, vi[u] - mi, st[2][u]);
      P.state[3 * n + k] = __fmaf_rn(dj, vj[u] - mj, st[3][u]);
      P.state[4 * n + k] = __fmaf_rn(di, vj[u] - mj, st[4][u]);
    }
  }
}
template <typename Source>
__global__ void __launch_bounds__(kThreads) pair_update_kernel(const __grid_constant__ Source pairs) {
  const NangilaPairDesc P = pairs.d[blockIdx.y];
  auto tile = [&](int64_t first) {
    if (P.dtype == NANGILA_F32) pair_tile<float>(P, first);
    else if (P.dtype == NANGILA_BF16) pair_tile<__nv_bfloat16>(P, first);
    else pair_tile<__half>(P, first);
  };
  const int64_t first = int64_t(blockIdx.x) * kPairTile + threadIdx.x;
  // Descriptors in device memory come with the caller's word for the largest pair, which may be too small: then a CTA takes more tiles. (Not in
  // the other form, whose grid is known to cover every pair: the loop takes the step of eight 589 824-element layers from 178 to 222 us.)
  if constexpr (Source::kGridMayBeShort) {
    for (int64_t f = first; f < P.numel; f += int64_t(gridDim.x) * kPairTile) tile(f);
  } else {
    tile(first);
  }
}

// out per pair (8 doubles): sum corr, valid corr, sum alpha(i->j), sum beta(i->j), valid(i->j),
//                           sum alpha(j->i), sum beta(j->i), valid(j->i)
__global__ void __launch_bounds__(kThreads) pair_finalize_kernel(const NangilaPairDesc* __restrict__ pairs, double* out) {
  __shared__ double sh[kThreads / 32];
  const NangilaPairDesc P = pairs[blockIdx.y];
  const float* mean_i = P.state;
  const float* mean_j = P.state + P.numel;
  const float* m2_i = P.state + 2 * P.numel;
  const float* m2_j = P.state + 3 * P.numel;
  const float* co = P.state + 4 * P.numel;
  const double denom = double(P.count_after > 1 ? P.count_after - 1 : 1);
  double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int64_t k = int64_t(blockIdx.x) * kThreads + threadIdx.x; k < P.numel; k += int64_t(gridDim.x) * kThreads) {
    const double vi = m2_i[k] / denom, vj = m2_j[k] / denom, cov = co[k] / denom;
    const double d = sqrt(vi * vj);
    if (d > 1e-10) {
      a[0] += cov / d;
      a[1] += 1.0;
    }
    if (vi > 1e-10) {  // i drives j
      const double al = cov / vi;
      a[2] += al;
      a[3] += double(mean_j[k]) - al * double(mean_i[k]);
      a[4] += 1.0;
    }
    if (vj > 1e-10) {  // j drives i
      const double al = cov / vj;
      a[5] += al;
      a[6] += double(mean_i[k]) - al * double(mean_j[k]);
      a[7] += 1.0;
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const double s = block_sum(a[q], sh);
    if (threadIdx.x == 0 && s != 0.0) atomicAdd(&out[blockIdx.y * 8 + q], s);
  }
}

int grid_x_for(int64_t max_numel) {
  int64_t b = (max_numel + kThreads * 4 - 1) / (kThreads * 4);
  return int(b < 1 ? 1 : (b > 148 * 4 ? 148 * 4 : b));
}

}  // namespace
}  // namespace nangila

namespace nangila {
namespace {
template <typename Source>
cudaError_t launch_sumsq(const Source& src, int count, int64_t max_numel, double* out, cudaStream_t stream) {
  const int64_t steps = (max_numel + kSumStep - 1) / kSumStep;
  const dim3 grid(unsigned(steps < 1 ? 1 : (steps > 148 * 4 ? 148 * 4 : steps)), unsigned(count));
  layer_sumsq_kernel<Source><<<grid, kThreads, 0, stream>>>(src, out);
  return cudaGetLastError();
}
template <typename Source>
cudaError_t launch_pairs(const Source& src, int count, int64_t max_numel, cudaStream_t stream) {
  const int64_t tiles = (max_numel + kPairTile - 1) / kPairTile;
  if (!Source::kGridMayBeShort && tiles > 0x7fffffffll) return cudaErrorInvalidValue;
  const dim3 grid(unsigned(tiles < 1 ? 1 : tiles > 0x7fffffffll ? 0x7fffffffll : tiles), unsigned(count));
  pair_update_kernel<Source><<<grid, kThreads, 0, stream>>>(src);
  return cudaGetLastError();
}
}  // namespace
}  // namespace nangila

// `layers` / `pairs` are DEVICE arrays of descriptors, or HOST arrays in the functions ending in _host (copied into the launch);
// `out` must be zero-filled by the caller.
extern "C" int nangila_sculptor_layer_sumsq(const NangilaLayerDesc* layers, int32_t nlayers, int64_t max_numel,
                                            double* out, cudaStream_t stream) {
  using namespace nangila;
  if (layers == nullptr || out == nullptr || nlayers <= 0 || nlayers > 65535) return int(cudaErrorInvalidValue);
  return int(launch_sumsq(FromMemory<NangilaLayerDesc>{layers}, nlayers, max_numel, out, stream));
}
extern "C" int nangila_sculptor_layer_sumsq_host(const NangilaLayerDesc* layers, int32_t nlayers, double* out, cudaStream_t stream) {
  using namespace nangila;
  using Source = FromParams<NangilaLayerDesc>;
  if (layers == nullptr || out == nullptr || nlayers <= 0 || nlayers > 65535) return int(cudaErrorInvalidValue);
  for (int i = 0; i < nlayers; i += Source::kMax) {
    Source src{};
    const int count = nlayers - i < Source::kMax ? nlayers - i : Source::kMax;
    int64_t mx = 1;
    for (int k = 0; k < count; ++k) {
      src.d[k] = layers[i + k];
      mx = layers[i + k].numel > mx ? layers[i + k].numel : mx;
    }
    const cudaError_t e = launch_sumsq(src, count, mx, out + i, stream);
    if (e != cudaSuccess) return int(e);
  }
  return 0;
}
extern "C" int nangila_sculptor_pair_update(const NangilaPairDesc* pairs, int32_t npairs, int64_t max_numel,
                                            cudaStream_t stream) {
  using namespace nangila;
  if (pairs == nullptr || npairs <= 0 || npairs > 65535) return int(cudaErrorInvalidValue);
  return int(launch_pairs(FromMemory<NangilaPairDesc>{pairs}, npairs, max_numel, stream));
}
extern "C" int nangila_sculptor_pair_update_host(const NangilaPairDesc* pairs, int32_t npairs, cudaStream_t stream) {
  using namespace nangila;
  using Source = FromParams<NangilaPairDesc>;
  if (pairs == nullptr || npairs <= 0 || npairs > 65535) return int(cudaErrorInvalidValue);
  for (int i = 0; i < npairs; i += Source::kMax) {
    Source src{};
    const int count = npairs - i < Source::kMax ? npairs - i : Source::kMax;
    int64_t mx = 1;
    for (int k = 0; k < count; ++k) {
      src.d[k] = pairs[i + k];
      mx = pairs[i + k].numel > mx ? pairs[i + k].numel : mx;
    }
    const cudaError_t e = launch_pairs(src, count, mx, stream);
    if (e != cudaSuccess) return int(e);
  }
  return 0;
}
extern "C" int nangila_sculptor_pair_finalize(const NangilaPairDesc* pairs, int32_t npairs, int64_t max_numel,
                                              double* out, cudaStream_t stream) {
  if (pairs == nullptr || out == nullptr || npairs <= 0 || npairs > 65535) return int(cudaErrorInvalidValue);
  dim3 grid(unsigned(nangila::grid_x_for(max_numel)), unsigned(npairs));
  nangila::pair_finalize_kernel<<<grid, nangila::kThreads, 0, stream>>>(pairs, out);
  return int(cudaGetLastError());
}
