// Quantizing parameter all-gather for fully-sharded training (sm_100a): every rank quantizes its
// parameter shard to INT8 (default) or INT4 with one bf16 scale per 64 elements, stores the codes
// straight into every other rank's staging slots over NVLink, and every rank dequantizes the shards
// straight into the unsharded parameter buffer the next layer reads. 1.03 (INT8) or 0.53 (INT4) bytes per
// element cross the links instead of 2.
//
// The owner of a shard also consumes the dequantized form of its own shard, so all ranks compute
// with bit-identical parameters. Rounding is to nearest (parameters must not pick up random noise).
//
// One behind the other: ag_quantize (codes to the peers, this rank's own part of the result; it may be the
// buffer the shard is read from), the meeting of the ranks (a kernel, or the start of the next one: meet.cuh), ag_expand (the other ranks' parts). Grids of short CTAs
// without flags or fences that the hardware hands out as SMs come free.
// What bounds them: HBM and L2 traffic. Measured on B200, four ranks on one device, 3.1 M bf16 elements each, INT8 (25 MB in, 39 MB of codes, 100 MB
// out): 17 us (5.2 TB/s) + 21 us (5.5 TB/s), 42.4 us for the call; as one resident kernel with block barriers and a flag per chunk 49.3 us.
// The arithmetic is kept out of the way: with divisions by the chunk size, conversions and clamps the two took 19 and 45 us (now 167 and 51 instructions per
// eight elements, the stores to three peers and this rank's own part among them).
//
// The reference leaves the FSDP parameter all-gather untouched (python/nangila/fsdp.py:80-236 only
// hooks the gradient path).
//
// Staging slots are double-buffered by launch parity: a rank may start launch t+1 while a slower
// peer still dequantizes launch t, but it cannot finish t+1 (and so cannot start t+2) before that
// peer has started t+1, because it needs the peer's word of t+1.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "fsdp_grid.cuh"
#include "meet.cuh"
#include "nangila_kernels.h"
#include "quant.cuh"
#include "signal.cuh"

namespace nangila {
namespace {

using namespace dev;
using namespace comm;

constexpr int kThreads = 256;
constexpr int kE = 8;
constexpr int kPerIter = kThreads * kE;  // 2048

__host__ __device__ inline uint64_t ag_slot_bytes(int chunk, int bits) {
  return uint64_t(chunk) * bits / 8 + uint64_t(chunk) / kQuantBlock * 2;
}

// eight values as they lie in memory
template <typename T>
struct __align__(16) Raw {
  T v[kE];
};
template <int BITS>
using Packed = std::conditional_t<BITS == 8, uint2, uint32_t>;  // eight codes

constexpr int kTile = 4;  // iterations of 2048 elements whose loads are issued together
// A small shard is quantized in tiles of one iteration: a CTA's four, one behind the other, are then what the call waits for. us a call, tiles of four / of
// one: 131 072 elements, one rank of eight, bf16 8.3 / 6.9, fp32 10.3 / 8.2; four emulated ranks of as many fp32 elements (256 CTAs) 10.1 / 8.3,
// of twice as many 11.3 / 12.9.
constexpr int64_t kSmallCtas = 2 * 148;

// A rank's shard in the exchange region: its codes one behind the other, then its scales. Worked out on the host: the number of chunks is a
// division of 64-bit numbers, which costs a thread more than quantizing eight elements.
struct AgShape {
  uint64_t base, per_owner, to_scales;
  AgShape(const NangilaAgParams& p, int bits) {
    const int C = p.chunk_elems;
    const uint64_t cps = uint64_t((p.shard_elems + C - 1) / C);
    per_owner = cps * ag_slot_bytes(C, bits);
    base = p.recv_off + uint64_t(p.epoch & 1u) * uint64_t(p.world) * per_owner;
    to_scales = cps * uint64_t(C) * uint64_t(bits) / 8;
  }
};
// Offsets of lane `tid` of iteration `it`; the next iterations follow kThreads lanes, kPerIter / 64 scales further.
template <int BITS>
struct AgSlot {
  uint64_t codes, scales;
  __device__ __forceinline__ AgSlot(const AgShape& sh, int owner, int it, int tid) {
    const uint64_t own = sh.base + uint64_t(owner) * sh.per_owner;
    codes = own + (uint64_t(it) * kPerIter + tid * kE) * BITS / 8;
    scales = own + sh.to_scales + (uint64_t(it) * (kPerIter / kQuantBlock) + tid / 8) * 2;
  }
};

// Eight values from their codes. For bf16 in packed arithmetic: a code and a scale have 8 significant bits, so their product is rounded
// once either way.
template <typename T, int BITS>
__device__ __forceinline__ void expand8(const Packed<BITS>& w, uint16_t scale, T* dst) {
  if constexpr (std::is_same_v<T, __nv_bfloat16>) {
    const uint32_t bits = scale;
    const bf162 s2 = as_bf162(bits | (bits << 16));
    bf162 q[4];
    if constexpr (BITS == 8) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // 0x43nn: 128 + the low seven bits, less 128 or (code below zero) 256
        const uint32_t v = __byte_perm(j < 2 ? w.x : w.y, 0x43434343u, (j & 1) == 0 ? 0x4140 : 0x4342);
        q[j] = __hsub2(as_bf162(v & 0xff7fff7fu), as_bf162(v & 0xff80ff80u));
      }
    } else {
      codes8_bf16(w, q);
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(as_u32(__hmul2(q[0], s2)), as_u32(__hmul2(q[1], s2)), as_u32(__hmul2(q[2], s2)), as_u32(__hmul2(q[3], s2)));
  } else {
    const float s = bf16_bits_to_float(scale);
    float y[kE];
#pragma unroll
    for (int i = 0; i < kE; ++i) {
      // the code plus 128 (or 8) as the low bits of a float near 2^23: one permutation and one exact subtraction, no conversion
      if constexpr (BITS == 8) y[i] = (__uint_as_float(__byte_perm((i < 4 ? w.x : w.y) ^ 0x80808080u, 0x4B000000u, 0x7440u + uint32_t(i & 3))) - 8388736.0f) * s;
      else y[i] = (__uint_as_float((((w ^ 0x88888888u) >> (4 * i)) & 0xfu) | 0x4B000000u) - 8388616.0f) * s;
    }
    Vec8<T>::store(dst, y);
  }
}

template <typename T, int BITS, int TILE>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 4 ? 4 : 5) ag_quantize_kernel(const __grid_constant__ NangilaAgParams p, const __grid_constant__ AgShape sh) {
  may_follow();
  const int vr = blockIdx.y, me = p.rank0 + vr, W = p.world, tid = threadIdx.x;
  const int total = int((p.shard_elems + kPerIter - 1) / kPerIter);
  // A rank that has failed does nothing more. The word is looked at when the first data are there, so it costs no latency.
  const uint32_t failed = *reinterpret_cast<volatile uint32_t*>(&p.status[vr][kStatusCode]);
  const T* in = static_cast<const T*>(p.in_shard[vr]);
  T* own = static_cast<T*>(p.out_full[vr]) + int64_t(me) * p.shard_elems;  // may be `in`: a lane writes where it has read
  constexpr float kInvQmax = BITS == 8 ? 0.0078740157f : 0.14285715f;
  for (int it0 = blockIdx.x * TILE; it0 < total; it0 += gridDim.x * TILE) {
    const int64_t at0 = int64_t(it0) * kPerIter + tid * kE, left = p.shard_elems - at0;  // the shard is a multiple of 8: a lane has eight values or none
    Raw<T> raw[TILE];
#pragma unroll
    for (int b = 0; b < TILE; ++b) raw[b] = b * kPerIter < left ? *reinterpret_cast<const Raw<T>*>(in + at0 + b * kPerIter) : Raw<T>{};
    if (failed != 0u) return;
    Packed<BITS> w[TILE];
    uint16_t sb[TILE];
#pragma unroll
    for (int b = 0; b < TILE; ++b) {
      float x[kE], amax = 0.0f;
      bool clean = false;
      if constexpr (std::is_same_v<T, __nv_bfloat16>) {
        const uint4 v = *reinterpret_cast<const uint4*>(&raw[b]);
        const uint32_t words[4] = {v.x, v.y, v.z, v.w};
        words_to_float8(words, x);
        clean = !__any_sync(0xffffffffu, maybe_nonfinite8(words));
        if (clean) amax = absmax8_bf16(words);
      } else {
        Vec8<T>::load(reinterpret_cast<const T*>(&raw[b]), x);
      }
      if (!clean) {
#pragma unroll
        for (int i = 0; i < kE; ++i) {
          x[i] = sanitize(x[i]);
          amax = fmaxf(amax, fabsf(x[i]));
        }
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
      const uint32_t scale = bf16_ceil_bits(__fmul_rn(amax, kInvQmax));
      const float s = bf16_bits_to_float(scale);
      const bool live = s > 1e-30f;
      const float inv = live ? __frcp_rn(s) : 0.0f;
      sb[b] = uint16_t(live ? scale : 0u);
      // To the nearest integer, ties to even, by adding 1.5 2^23: the code is in the low bits (conversions run at a quarter of the rate).
      // The scale is rounded up, so that |x / s| stays below 127.5 (7.5) and needs no clamp.
      uint32_t q[kE];
#pragma unroll
      for (int i = 0; i < kE; ++i) q[i] = __float_as_uint(__fadd_rn(__fmul_rn(x[i], inv), 12582912.0f));
      const uint32_t lo = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
      const uint32_t hi = __byte_perm(__byte_perm(q[4], q[5], 0x0040), __byte_perm(q[6], q[7], 0x0040), 0x5410);
      if constexpr (BITS == 8) {
        w[b] = make_uint2(lo, hi);
      } else {
        const uint32_t a = lo & 0x0F0F0F0Fu, c = hi & 0x0F0F0F0Fu;
        w[b] = __byte_perm(a | (a >> 4), c | (c >> 4), 0x6420);
      }
    }
    const AgSlot<BITS> slot(sh, me, it0, tid);
    for (int d = 1, r = me + 1; d < W; ++d, ++r) {
      if (r == W) r = 0;
      Packed<BITS>* codes = reinterpret_cast<Packed<BITS>*>(p.region[r] + slot.codes);
      uint16_t* scales = reinterpret_cast<uint16_t*>(p.region[r] + slot.scales);
#pragma unroll
      for (int b = 0; b < TILE; ++b) {
        if (it0 + b < total) {
          codes[b * kThreads] = w[b];
          if ((tid & 7) == 0) scales[b * (kPerIter / kQuantBlock)] = sb[b];
        }
      }
    }
    // this rank's own part of the result: what the others make of the codes
#pragma unroll
    for (int b = 0; b < TILE; ++b)
      if (b * kPerIter < left) expand8<T, BITS>(w[b], sb[b], own + at0 + b * kPerIter);
  }
}

template <typename T, int BITS, Met MET, bool ALL>  // ALL: there are fewer CTAs than owners, so one takes several of these
__global__ void __launch_bounds__(kThreads, MET == kMetBefore ? 8 : 4) ag_expand_kernel(const __grid_constant__ NangilaAgParams p, const __grid_constant__ AgShape sh, int tiles) {
  const int vr = blockIdx.z, me = p.rank0 + vr, W = p.world, tid = threadIdx.x;
  follow();
  uint32_t seen;
  if (!arrive<MET>(p, vr, p.flag_off, kTimeoutPhase3, 3u, seen)) return;
  const uint8_t* myreg = p.region[me];
  int d = blockIdx.y;
  do {
    int o = me + 1 + d;  // the other ranks' shards
    if (o >= W) o -= W;
    T* __restrict__ out = static_cast<T*>(p.out_full[vr]) + int64_t(o) * p.shard_elems;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int64_t at0 = int64_t(tile) * (kTile * kPerIter) + tid * kE, left = p.shard_elems - at0;
      const AgSlot<BITS> slot(sh, o, tile * kTile, tid);
      const Packed<BITS>* codes = reinterpret_cast<const Packed<BITS>*>(myreg + slot.codes);
      const uint16_t* scales = reinterpret_cast<const uint16_t*>(myreg + slot.scales);
      Packed<BITS> w[kTile];
      uint16_t sc[kTile];
#pragma unroll
      for (int b = 0; b < kTile; ++b) {
        if (b * kPerIter < left) {
          w[b] = codes[b * kThreads];
          sc[b] = scales[b * (kPerIter / kQuantBlock)];
        }
      }
      if (!all_came<MET>(p, vr, seen, kTimeoutPhase3, 3u)) return;
#pragma unroll
      for (int b = 0; b < kTile; ++b)
        if (b * kPerIter < left) expand8<T, BITS>(w[b], sc[b], out + at0 + b * kPerIter);
    }
    d += gridDim.y;
  } while (ALL && d < W - 1);
}

template <typename T, int BITS>
cudaError_t launch(const NangilaAgParams& p, cudaStream_t stream) {
  const int64_t total = (p.shard_elems + kPerIter - 1) / kPerIter, tiles = (total + kTile - 1) / kTile;
  if (tiles > kMaxTiles) return cudaErrorInvalidValue;
  const AgShape sh(p, BITS);
  if (total * p.nvr <= kSmallCtas) ag_quantize_kernel<T, BITS, 1><<<dim3(fsdp_grid(total, 1, p.grid_x).x, unsigned(p.nvr)), kThreads, 0, stream>>>(p, sh);
  else ag_quantize_kernel<T, BITS, kTile><<<dim3(fsdp_grid(tiles, 1, p.grid_x).x, unsigned(p.nvr)), kThreads, 0, stream>>>(p, sh);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || p.world == 1) return e;
  const FsdpGrid g = fsdp_grid(tiles, p.world - 1, p.grid_x);
  const Met met = how_to_meet(p, int64_t(g.x) * g.y * p.nvr, 4 * 148);
  if ((e = launch_meet(p, met, p.flag_off, kTimeoutPhase3, 3u, stream)) != cudaSuccess) return e;
  auto* expand = met == kMetInLaunch ? ag_expand_kernel<T, BITS, kMetInLaunch, true> : met == kMeetHere ? ag_expand_kernel<T, BITS, kMeetHere, true>
                 : g.walk == kWalkGroups ? ag_expand_kernel<T, BITS, kMetBefore, true> : ag_expand_kernel<T, BITS, kMetBefore, false>;
  return launch_following(expand, dim3(g.x, g.y, unsigned(p.nvr)), kThreads, 0, stream, p, sh, int(tiles));
}

}  // namespace
}  // namespace nangila

extern "C" uint64_t nangila_ag_region_bytes(int64_t shard_elems, int32_t world, int32_t chunk_elems, int32_t bits,
                                            uint64_t* recv_off, uint64_t* flag_off) {
  auto align = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
  const uint64_t cps = uint64_t((shard_elems + chunk_elems - 1) / chunk_elems);
  uint64_t off = 0;
  if (recv_off) *recv_off = off;
  off = align(off + 2 * uint64_t(world) * cps * nangila::ag_slot_bytes(chunk_elems, bits));
  if (flag_off) *flag_off = off;
  off = align(off + uint64_t(world) * cps * 4);
  return off;
}

// Chunk size for a shard: what a rank's slot is rounded up to. About one chunk for each of the `resident`
// CTAs that a device holds at once per rank (NANGILA_LAYOUT_CTAS), not below 4096 elements except for shards of less than four
// such chunks. The same on every rank, whatever its device: peers write into one another's slots.
extern "C" int32_t nangila_ag_chunk_elems(int64_t shard_elems, int32_t resident) {
  const int64_t g = resident > 0 ? resident : 1, most = 131072;
  const int64_t waves = std::max<int64_t>(1, (shard_elems + g * most - 1) / (g * most));
  const int64_t per = (shard_elems + g * waves - 1) / (g * waves);
  const int64_t least = (shard_elems < 4 * 4096 ? 1 : 2) * nangila::kPerIter;
  return int32_t(std::min<int64_t>(most, std::max<int64_t>(least, (per + nangila::kPerIter - 1) / nangila::kPerIter * nangila::kPerIter)));
}

extern "C" int nangila_ag_launch(const NangilaAgParams* p, cudaStream_t stream) {
  using namespace nangila;
  if (p == nullptr || p->shard_elems <= 0 || p->shard_elems % 8 != 0 || p->world < 1 || p->world > NANGILA_MAX_RANKS ||
      p->nvr < 1 || p->nvr > NANGILA_MAX_VRANKS || p->rank0 < 0 || p->rank0 + p->nvr > p->world ||
      (p->nvr > 1 && p->nvr != p->world) || p->chunk_elems <= 0 || p->chunk_elems % kPerIter != 0 || p->epoch == 0 ||
      (p->bits != 8 && p->bits != 4))
    return int(cudaErrorInvalidValue);
  switch (p->dtype) {
    case NANGILA_F32: return int(p->bits == 8 ? launch<float, 8>(*p, stream) : launch<float, 4>(*p, stream));
    case NANGILA_BF16: return int(p->bits == 8 ? launch<__nv_bfloat16, 8>(*p, stream) : launch<__nv_bfloat16, 4>(*p, stream));
    case NANGILA_F16: return int(p->bits == 8 ? launch<__half, 8>(*p, stream) : launch<__half, 4>(*p, stream));
    default: return int(cudaErrorInvalidValue);
  }
}
