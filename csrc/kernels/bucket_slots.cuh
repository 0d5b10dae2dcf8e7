// Slot layout of the kernels that exchange block-INT4 chunks (predres_bucket.cu, fsdp_reduce_scatter.cu).
#pragma once
#include <cstdint>

#include "quant.cuh"

namespace nangila {
namespace dev {

constexpr int kThreads = 256;
constexpr int kE = kElems8;                       // elements per thread per iteration
constexpr int kElemsPerIter = kThreads * kE;      // 2048

// packed nibbles, then one bf16 scale per 64 elements, then a 16-byte trailer whose first word is the
// sender's prediction gain (phase 1) or the mean gain of all senders (phase 2)
__host__ __device__ inline uint64_t compressed_trailer_off(int chunk) {
  return uint64_t(chunk) / 2 + uint64_t(chunk) / kQuantBlock * 2;
}
__host__ __device__ inline uint64_t compressed_slot_bytes(int chunk) { return compressed_trailer_off(chunk) + 16; }

// Slot layout (compressed modes), warp-major so that everything one warp needs from a chunk is
// contiguous and can be fetched with one bulk copy: packed nibbles [warp][iteration][lane] (4 bytes per
// lane = 8 elements), then bf16 scales [warp][iteration][4] (one per 64 elements), then the trailer.
__device__ __forceinline__ uint32_t* packed_ptr(uint8_t* slot, int C, int it, int tid) {
  const int iters = C / kElemsPerIter;
  return reinterpret_cast<uint32_t*>(slot) + ((tid >> 5) * iters + it) * 32 + (tid & 31);
}
__device__ __forceinline__ uint16_t* scale_ptr(uint8_t* slot, int C, int it, int tid) {
  const int iters = C / kElemsPerIter;
  return reinterpret_cast<uint16_t*>(slot + uint64_t(C) / 2) + ((tid >> 5) * iters + it) * 4 + ((tid & 31) >> 3);
}

}  // namespace dev
}  // namespace nangila
