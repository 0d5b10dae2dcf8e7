// Compressed gradient reduce-scatter for fully-sharded training (sm_100a). Rank o owns shard o of the bucket (W equal shards, cut
// into chunks of chunk_elems). One behind the other:
//
//   rs_quantize   x = g + error memory, block-INT4 codes and scales of every chunk stored into the owner's slot [chunk][me] over
//                 NVLink, new error memory
//   meeting       every rank's codes are in place: a kernel of its own, or the start of the next one (meet.cuh)
//   rs_sum        the sum of the W contributions of this rank's shard times out_scale
//
// Grids of short CTAs without flags, fences or residency that the hardware hands out as SMs come free. Slots alternate between two sets
// by launch parity: a rank may start the next launch while a peer still sums, but it cannot get two launches ahead, because its meeting in
// between needs that peer's word.
//
// What bounds it: rs_quantize the issue rate, about as much as HBM (the gradient in), rs_sum latency (its input lies in L2). Measured on B200, four ranks on one
// device, 12.6 M bf16 elements each: 26 us (100 MB in, 27 MB of codes out: 4.8 TB/s) + 12 us, 43 us for the call; before, one resident kernel that walked a
// task per chunk with a ring of bulk copies, a fence and a flag each: 99 us. Tiles of four iterations: their loads are issued together,
// and the index arithmetic is paid once.
//
// Takes the place of the reference's FSDP hook (python/nangila/fsdp.py:107-236).
#include <algorithm>
#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "bucket_slots.cuh"
#include "fsdp_grid.cuh"
#include "fsdp_reduce_scatter.cuh"
#include "meet.cuh"
#include "nangila_kernels.h"
#include "quant.cuh"
#include "signal.cuh"

namespace nangila {
namespace {

using namespace dev;
using namespace comm;

// Iterations of 2048 elements a CTA takes; their loads are issued together.
constexpr int kTile = 4;

// What follows from the parameters, worked out once on the host: two of them are divisions of 64-bit numbers, which cost a thread more than
// quantizing eight elements (the call above: 45.2 us with them in every CTA).
struct RsShape {
  int W, C, iters, cps, sub, tiles;  // sub: tiles of a chunk; tiles: of a shard
  int64_t shard;
  uint64_t slot, recv;
  explicit RsShape(const NangilaPredResParams& p)
      : W(p.world), C(p.chunk_elems), iters(C / kElemsPerIter), cps(p.nchunks / p.world), sub((iters + kTile - 1) / kTile), tiles(cps * sub),
        shard(p.n / p.world), slot(compressed_slot_bytes(C)), recv(p.recv1_off + uint64_t(p.epoch & 1u) * uint64_t(cps) * W * slot) {}
};

// Packed-bf16 arithmetic where gradient and error memory are bf16, in chunks that lie wholly inside the shard.
template <typename T, typename S>
constexpr bool kPackedBf16 = std::is_same_v<T, __nv_bfloat16> && std::is_same_v<S, __nv_bfloat16>;

// (A loop's invariants cost registers; without one 64 are enough for four CTAs an SM. Packed bf16 without error memory: six, although 16 bytes a thread
// spill; without spills 43.0 us with five and 45.5 with four for the call above, against 42.8.)
template <typename T, typename S, bool EF, Walk WALK>
__global__ void __launch_bounds__(kThreads, WALK != kNoWalk ? 2 : kPackedBf16<T, S> && !EF ? 6 : 4) rs_quantize_kernel(const __grid_constant__ NangilaPredResParams p, const __grid_constant__ RsShape sh) {
  may_follow();
  const int vr = blockIdx.z, me = p.rank0 + vr, W = sh.W, C = sh.C, tid = threadIdx.x;
  // A rank that has failed does nothing more. The word is looked at when the first data are there, so it costs no latency.
  const uint32_t failed = *reinterpret_cast<volatile uint32_t*>(&p.status[vr][kStatusCode]);
  const T* __restrict__ grad = static_cast<const T*>(p.grad[vr]);
  S* __restrict__ ef = static_cast<S*>(p.ef[vr]);
  const bool has_ef = EF && ef != nullptr;
  const uint32_t key = make_key(p.seed, p.step, p.bucket_id, uint32_t(me), 1u);
  const bool stochastic = p.stochastic != 0;
  int d = blockIdx.y;
  do {
    int o = me + 1 + d;  // remote owners first, this rank's own shard last
    if (o >= W) o -= W;
    int tile = blockIdx.x;
    do {
      const int j = int(unsigned(tile) / unsigned(sh.sub)), it0 = (tile - j * sh.sub) * kTile;
      const int64_t first = int64_t(o) * sh.shard + int64_t(j) * C, limit = int64_t(o + 1) * sh.shard;
      const bool whole = first + C <= limit;
      uint8_t* dst = p.region[o] + sh.recv + (uint64_t(j) * W + me) * sh.slot;
      const int64_t at0 = first + int64_t(it0) * kElemsPerIter + tid * kE;  // this lane's first element
      const int left = min(kTile, sh.iters - it0);                          // iterations of this tile
      const T* g0 = grad + at0;
      S* e0 = ef + at0;  // (not used where there is no error memory)
      uint32_t* codes = packed_ptr(dst, C, it0, tid);
      uint16_t* scales = scale_ptr(dst, C, it0, tid);
      auto put = [&](int b, uint32_t packed, uint32_t scale) {
        codes[b * 32] = packed;
        if ((tid & (kLanes8 - 1)) == 0) scales[b * 4] = uint16_t(scale);
      };
      // eight values in FP32; e: the error memory
      auto fp32 = [&](auto guard, int b, float (&g)[kE], float (&e)[kE]) {
        constexpr bool GUARD = decltype(guard)::value;
#pragma unroll
        for (int i = 0; i < kE; ++i) e[i] = has_ef ? e[i] + sanitize(g[i]) : sanitize(g[i]);
        uint32_t packed, scale;
        quantize8(e, key, uint32_t((at0 + b * kElemsPerIter) >> 1), stochastic, packed, scale);
        if (has_ef) store8<S, GUARD>(e0, b * kElemsPerIter, limit - at0, e);
        put(b, packed, scale);
      };
      auto fp32_tile = [&](auto guard) {
        constexpr bool GUARD = decltype(guard)::value;
        constexpr int kBatch = 2;
#pragma unroll 1
        for (int b0 = 0; b0 < left; b0 += kBatch) {
          float g[kBatch][kE], e[kBatch][kE];
#pragma unroll
          for (int b = 0; b < kBatch; ++b)
            if (b0 + b < left) {
              load8<T, GUARD>(g0, (b0 + b) * kElemsPerIter, limit - at0, g[b]);
              if (has_ef) load8<S, GUARD>(e0, (b0 + b) * kElemsPerIter, limit - at0, e[b]);
            }
          if (failed != 0u) return;
#pragma unroll
          for (int b = 0; b < kBatch; ++b)
            if (b0 + b < left) fp32(guard, b0 + b, g[b], e[b]);
        }
      };
      if (!whole) {
        fp32_tile(std::true_type{});
      } else if constexpr (kPackedBf16<T, S>) {
        uint4 g[kTile], e[kTile];
#pragma unroll
        for (int b = 0; b < kTile; ++b) {
          if (b < left) {
            g[b] = *reinterpret_cast<const uint4*>(g0 + b * kElemsPerIter);
            if (has_ef) e[b] = *reinterpret_cast<const uint4*>(e0 + b * kElemsPerIter);
          }
        }
        if (failed != 0u) return;
#pragma unroll
        for (int b = 0; b < kTile; ++b) {
          if (b >= left) break;
          const uint32_t gw[4] = {g[b].x, g[b].y, g[b].z, g[b].w}, ew[4] = {e[b].x, e[b].y, e[b].z, e[b].w};
          uint32_t x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] = has_ef ? as_u32(__hadd2(as_bf162(gw[k]), as_bf162(ew[k]))) : gw[k];
          if (__any_sync(0xffffffffu, maybe_nonfinite8(x))) {  // a NaN / Inf in the warp's slice (or magnitudes >= 2): sanitised in FP32
            float gf[kE], err[kE];
            words_to_float8(gw, gf);
            words_to_float8(ew, err);
            fp32(std::false_type{}, b, gf, err);
            continue;
          }
          uint32_t packed, scale, qs[4];
          quantize8_bf16(x, packed, scale, qs);
          if (has_ef) *reinterpret_cast<uint4*>(e0 + b * kElemsPerIter) = make_uint4(x[0], x[1], x[2], x[3]);
          put(b, packed, scale);
        }
      } else {
        fp32_tile(std::false_type{});
      }
      tile += gridDim.x;
    } while (WALK != kNoWalk && tile < sh.tiles);
    d += gridDim.y;
  } while (WALK == kWalkGroups && d < W);
}

template <typename T, bool PACKED, Met MET>
__global__ void __launch_bounds__(kThreads, 4) rs_sum_kernel(const __grid_constant__ NangilaPredResParams p, const __grid_constant__ RsShape sh) {
  const int vr = blockIdx.y, me = p.rank0 + vr, W = sh.W, C = sh.C, tid = threadIdx.x;
  uint8_t* myreg = p.region[me];
  follow();
  uint32_t seen;
  if (!arrive<MET>(p, vr, p.flag1_off, kTimeoutPhase2, 2u, seen)) return;
  T* __restrict__ out = static_cast<T*>(p.out_shard[vr]);
  for (int tile = blockIdx.x; tile < sh.tiles; tile += gridDim.x) {
    const int j = int(unsigned(tile) / unsigned(sh.sub)), it0 = (tile - j * sh.sub) * kTile;
    uint8_t* src = myreg + sh.recv + uint64_t(j) * W * sh.slot;
    const uint32_t* codes = packed_ptr(src, C, it0, tid);
    const uint16_t* scales = scale_ptr(src, C, it0, tid);
    const uint64_t to_scales = reinterpret_cast<const uint8_t*>(scales) - reinterpret_cast<const uint8_t*>(codes);
    const int left = min(kTile, sh.iters - it0);
    const int64_t at0 = int64_t(j) * C + int64_t(it0) * kElemsPerIter + tid * kE;
    // codes and scales of rank r for iterations b0 .. b0 + N - 1 of the tile
    auto fetch = [&](int r, int b0, auto& packed, auto& scale) {
      const uint8_t* from = reinterpret_cast<const uint8_t*>(codes) + uint64_t(r) * sh.slot;
      constexpr int N = sizeof(packed) / sizeof(packed[0]);
#pragma unroll
      for (int b = 0; b < N; ++b) {
        packed[b] = b0 + b < left ? reinterpret_cast<const uint32_t*>(from)[(b0 + b) * 32] : 0u;
        scale[b] = b0 + b < left ? reinterpret_cast<const uint16_t*>(from + to_scales)[(b0 + b) * 4] : uint16_t(0);
      }
    };
    if (PACKED && int64_t(j + 1) * C <= sh.shard) {
      // packed-bf16 form (quant.cuh): out_scale is folded into each rank's block scale, so the sum is already the result
      uint32_t acc[kTile][4] = {};
#pragma unroll 4
      for (int r = 0; r < W; ++r) {
        uint32_t packed[kTile];
        uint16_t scale[kTile];
        fetch(r, 0, packed, scale);
#pragma unroll
        for (int b = 0; b < kTile; ++b) {
          const float s = bf16_bits_to_float(scale[b]) * p.out_scale;
          dequant8_bf16_fma2(packed[b], __floats2bfloat162_rn(s, s), acc[b]);
        }
      }
      if (!all_came<MET>(p, vr, seen, kTimeoutPhase2, 2u)) return;
#pragma unroll
      for (int b = 0; b < kTile; ++b)
        if (b < left) *reinterpret_cast<uint4*>(out + at0 + b * kElemsPerIter) = make_uint4(acc[b][0], acc[b][1], acc[b][2], acc[b][3]);
    } else {
      constexpr int kBatch = 2;
#pragma unroll 1
      for (int b0 = 0; b0 < left; b0 += kBatch) {
        float acc[kBatch][kE] = {};
#pragma unroll 4
        for (int r = 0; r < W; ++r) {
          uint32_t packed[kBatch];
          uint16_t scale[kBatch];
          fetch(r, b0, packed, scale);
#pragma unroll
          for (int b = 0; b < kBatch; ++b) dequant8_add(packed[b], bf16_bits_to_float(scale[b]), acc[b]);
        }
        if (!all_came<MET>(p, vr, seen, kTimeoutPhase2, 2u)) return;
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
          if (b0 + b < left) {
#pragma unroll
            for (int i = 0; i < kE; ++i) acc[b][i] *= p.out_scale;
            store8_guarded<T>(out, at0 + (b0 + b) * kElemsPerIter, sh.shard, acc[b]);
          }
      }
    }
  }
}

template <typename T, typename S, bool EF>
void launch_quantize(const NangilaPredResParams& p, const RsShape& sh, cudaStream_t stream) {
  const FsdpGrid g = fsdp_grid(sh.tiles, p.world, p.grid_x);
  const dim3 grid(g.x, g.y, unsigned(p.nvr));
  if (g.walk == kNoWalk) rs_quantize_kernel<T, S, EF, kNoWalk><<<grid, kThreads, 0, stream>>>(p, sh);
  else if (g.walk == kWalkTiles) rs_quantize_kernel<T, S, EF, kWalkTiles><<<grid, kThreads, 0, stream>>>(p, sh);
  else rs_quantize_kernel<T, S, EF, kWalkGroups><<<grid, kThreads, 0, stream>>>(p, sh);
}

template <typename T, typename S>
cudaError_t launch(const NangilaPredResParams& p, cudaStream_t stream) {
  const int64_t sub = (p.chunk_elems / kElemsPerIter + kTile - 1) / kTile, all = p.nchunks / p.world * sub;
  if (all > kMaxTiles) return cudaErrorInvalidValue;
  const RsShape sh(p);
  const int phases = (p.phase_mask & 7) == 0 ? 7 : p.phase_mask;
  if (phases & 1) {
    bool ef = false;
    for (int v = 0; v < p.nvr; ++v) ef = ef || p.ef[v] != nullptr;
    if (ef) launch_quantize<T, S, true>(p, sh, stream);
    else launch_quantize<T, S, false>(p, sh, stream);
  }
  if (phases & 2) {
    cudaError_t e = cudaGetLastError();
    const dim3 grid(fsdp_grid(sh.tiles, 1, p.grid_x).x, unsigned(p.nvr));
    const Met met = how_to_meet(p, int64_t(grid.x) * grid.y, 8 * 148);
    if (e == cudaSuccess) e = launch_meet(p, met, p.flag1_off, kTimeoutPhase2, 2u, stream);
    if (e != cudaSuccess) return e;
    constexpr bool PACKED = kPackedBf16<T, S>;
    auto* sum = met == kMetBefore ? rs_sum_kernel<T, PACKED, kMetBefore> : met == kMetInLaunch ? rs_sum_kernel<T, PACKED, kMetInLaunch> : rs_sum_kernel<T, PACKED, kMeetHere>;
    return launch_following(sum, grid, kThreads, 0, stream, p, sh);
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_reduce_scatter(const NangilaPredResParams& p, cudaStream_t stream) {
  const bool s32 = p.state_dtype == NANGILA_F32;
  switch (p.grad_dtype) {
    case NANGILA_F32: return s32 ? launch<float, float>(p, stream) : launch<float, __nv_bfloat16>(p, stream);
    case NANGILA_BF16: return s32 ? launch<__nv_bfloat16, float>(p, stream) : launch<__nv_bfloat16, __nv_bfloat16>(p, stream);
    case NANGILA_F16: return s32 ? launch<__half, float>(p, stream) : launch<__half, __nv_bfloat16>(p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace nangila

extern "C" int32_t nangila_fsdp_grid(int64_t tiles, int32_t groups, int32_t cap, uint32_t* x, uint32_t* y) {
  const nangila::FsdpGrid g = nangila::fsdp_grid(tiles, groups, cap);
  *x = g.x;
  *y = g.y;
  return int32_t(g.walk);
}

// The slots of both parities and the flag words (one per rank is used; a region has room for one per chunk).
extern "C" uint64_t nangila_rs_region_bytes(int64_t n, int32_t world, int32_t chunk_elems, uint64_t* recv1_off,
                                            uint64_t* flag1_off, int32_t* nchunks) {
  auto align = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
  const int64_t shard = n / world;
  const uint64_t cps = uint64_t((shard + chunk_elems - 1) / chunk_elems);
  if (nchunks) *nchunks = int32_t(cps * world);
  uint64_t off = 0;
  if (recv1_off) *recv1_off = off;
  off = align(off + 2 * cps * world * nangila::dev::compressed_slot_bytes(chunk_elems));
  if (flag1_off) *flag1_off = off;
  off = align(off + cps * world * 4);
  return off;
}
