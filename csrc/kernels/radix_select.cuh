// Pieces of the three-pass radix select over the bit pattern of |x| (bits [30:20], [19:9], [8:0])
// shared by the DGC kernel and the absmax / percentile kernel.
#pragma once
#include <cstdint>

namespace nangila {
namespace rsel {

constexpr int kBins0 = 2048, kBins1 = 2048, kBins2 = 512;

// Scanning bins from the top, find the bin that holds the `want`-th largest element (1-based) and
// reduce `want` to the rank inside that bin; bin 0 if there are fewer elements. All 256 threads of the CTA take part: thread t owns
// the t-th stretch of bins from the top, a block-wide prefix sum finds the stretch, its owner the bin. (One warp walking down 32 bins
// at a time waits for L2 at every step: 20 us for a value near 1, whose bin is in the middle; this takes about 1.5.)
// `sh` is 10 words of shared memory. `hist` must be complete (grid barrier before the call).
template <int NBINS>
__device__ inline void select_bin(const uint32_t* hist, uint32_t& want, uint32_t& bin, uint32_t* sh) {
  constexpr int kPer = NBINS / 256;
  static_assert(NBINS % 256 == 0, "whole stretches");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int top = NBINS - 1 - tid * kPer;  // highest bin of this thread
  uint32_t c[kPer], mine = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    c[i] = __ldcg(hist + top - i);
    mine += c[i];
  }
  uint32_t incl = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) sh[warp] = incl;
  if (tid == 0) sh[8] = 0u;
  __syncthreads();
  uint32_t before = incl - mine, all = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) before += sh[w];
    all += sh[w];
  }
  if (before < want && want <= before + mine) {
    uint32_t rest = want - before;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (rest > 0 && rest <= c[i]) {
        sh[8] = uint32_t(top - i);
        sh[9] = rest;
        rest = 0;
      } else if (rest > 0) {
        rest -= c[i];
      }
    }
  } else if (tid == 0 && want > all) {
    sh[9] = want - all;
  }
  __syncthreads();
  bin = sh[8];
  want = sh[9];
  __syncthreads();
}

}  // namespace rsel
}  // namespace nangila
