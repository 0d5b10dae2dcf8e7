// Pieces of the three-pass radix select over the bit pattern of |x| (bits [30:20], [19:9], [8:0])
// shared by the DGC kernel and the absmax / percentile kernel.
#pragma once
#include <cstdint>

namespace nangila {
namespace rsel {

constexpr int kBins0 = 2048, kBins1 = 2048, kBins2 = 512;

// Scanning bins from the top, find the bin that holds the `want`-th largest element (1-based) and
// reduce `want` to the rank inside that bin; bin 0 if there are fewer elements. All 256 threads of the CTA take part: warp w owns the
// w-th stretch of bins from the top and reads it four bins a lane, neighbouring lanes neighbouring groups; prefix sums find the group.
// `sh` is 10 words of shared memory. `hist` must be complete (grid barrier before the call).
//
// Bound by L2: every CTA of a grid reads the same few kilobytes at the same time. With a lane on a stretch of its own, word by word, a
// warp's load touched 32 sectors: 444 CTAs took 12 us for 4096 bins and 5 for 2048. Read as whole lines they
// take under 2 each, and the DGC step of 13.1 M entries 73 us instead of 87.
template <int NBINS>
__device__ inline void select_bin(const uint32_t* hist, uint32_t& want, uint32_t& bin, uint32_t* sh) {
  static_assert(NBINS % 512 == 0, "whole lines");
  constexpr int kGroups = NBINS / 4, kRounds = (kGroups + 255) / 256;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool vec = (reinterpret_cast<uintptr_t>(hist) & 15u) == 0;  // wherever the caller's words lie
  uint32_t c[kRounds][4], upto[kRounds], mine = 0;  // bins of a group from the top; entries of this warp's stretch up to and with the group
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    const int g = (warp * kRounds + i) * 32 + lane;  // from the top
    const uint32_t* at = hist + NBINS - 4 - 4 * g;
#pragma unroll
    for (int k = 0; k < 4; ++k) c[i][k] = 0u;
    if (g < kGroups) {
      if (vec) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(at));
        c[i][0] = v.w; c[i][1] = v.z; c[i][2] = v.y; c[i][3] = v.x;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) c[i][k] = __ldcg(at + 3 - k);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    uint32_t incl = c[i][0] + c[i][1] + c[i][2] + c[i][3];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    upto[i] = mine + incl;
    mine += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 31) sh[warp] = mine;
  if (tid == 0) sh[8] = 0u;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) before += sh[w];
    all += sh[w];
  }
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    const uint32_t end = before + upto[i], begin = end - (c[i][0] + c[i][1] + c[i][2] + c[i][3]);
    if (begin < want && want <= end) {  // one group at most
      uint32_t rest = want - begin;
      const int top = NBINS - 1 - 4 * ((warp * kRounds + i) * 32 + lane);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (rest > 0 && rest <= c[i][k]) {
          sh[8] = uint32_t(top - k);
          sh[9] = rest;
          rest = 0;
        } else if (rest > 0) {
          rest -= c[i][k];
        }
      }
    }
  }
  if (tid == 0 && want > all) sh[9] = want - all;
  __syncthreads();
  bin = sh[8];
  want = sh[9];
  __syncthreads();
}

}  // namespace rsel
}  // namespace nangila
