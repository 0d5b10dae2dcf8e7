// Device-side packet codec: the prediction-residual compressor of the host core
// (csrc/core/compressor.hpp, PredictionResidualCompressor) for a tensor that lives on the GPU, writing
// and reading the host's own wire format, so a packet made on the device decodes on the host and the
// other way round:
//
//   payload = f32 -64 (block size, negated) | u32 numel | u32 ndim = 1 | u32 numel | f32 kappa |
//             f32 scale[ceil(numel / 64)] | u8 packed[ceil(numel / 2)]   (low nibble = even element)
//
// Three kernels: the two inner products that give the least-squares prediction gain
// kappa = clip(<g + ef, g_hat> / <g_hat, g_hat>, 0, 1); the encoder (x = g + ef - kappa g_hat, one FP32
// scale per 64 elements = amax / 7, round to nearest, error memory, nibble packing); the decoder
// (out = q * scale + kappa g_hat). kappa stays on the device between the first two, so nothing
// synchronises. This is what NangilaHook.compress_gpu / decompress_gpu and the C entry points
// nangila_compress_gpu / nangila_decompress_gpu run (reference: nangila-hook/src/python.rs:315-460 and
// ffi.rs:526-840, whose versions launched predict.cu / reconstruct.cu with one scale per tensor).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "nangila_kernels.h"
#include "quant.cuh"

namespace nangila {
namespace {

using namespace dev;

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 1184;  // grid-stride loops: enough blocks to fill any current device
constexpr int kPer = 8;  // elements per thread and iteration: one packed word, one eighth of a scale block
constexpr int kTile = kThreads * kPer;
// The encoder walks a tensor from its end, where the gains before it have just been, and the decoder from its start, where the encoder has ended: each
// begins with what the pass before it has left in L2, and what is not read again is marked to go first. (The order of the gains' sums, and so
// their rounding, stays as it was.) Measured on B200, 38.6 M bf16 elements: encoder 112 -> 107 us.
__host__ __device__ __forceinline__ int64_t tiles_of(int64_t n) { return (n + kTile - 1) / kTile; }

// LAST: nobody reads these again soon.
template <bool LAST = false, typename T>
__device__ __forceinline__ void load8_any(const T* p, int64_t base, int64_t n, float (&v)[8]) {
  // the tensor may start at any element-aligned address: vector loads only when 16-byte aligned
  if (base + 8 <= n && ((reinterpret_cast<uintptr_t>(p + base) & 15u) == 0)) {
    if constexpr (LAST) {
      uint4 w[sizeof(T) / 2];
#pragma unroll
      for (int i = 0; i < int(sizeof(T) / 2); ++i) w[i] = __ldcs(reinterpret_cast<const uint4*>(p + base) + i);
      Vec8<T>::load(reinterpret_cast<const T*>(w), v);
    } else {
      Vec8<T>::load(p + base, v);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (base + i < n) ? Vec16<T>::to_float(p[base + i]) : 0.0f;
  }
}
template <bool LAST = false>
__device__ __forceinline__ void load8_f32(const float* p, int64_t base, int64_t n, float (&v)[8]) {
  if (p == nullptr) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    return;
  }
  load8_any<LAST>(p, base, n, v);
}

// Eight values from `base` on; as with the loads, two 16-byte stores where the address allows it (a warp's two stores
// together fill whole lines; eight 4-byte stores per lane were 32-byte strided and took the decoder to 2.6 TB/s. Measured
// on B200 at 38.6 M elements: decoder 183 -> 83 us, 5.8 TB/s; encoder, bf16 gradient, 134 -> 120 us, 6.0 TB/s).
template <bool LAST = false>
__device__ __forceinline__ void store8_f32(float* p, int64_t base, int64_t n, const float (&v)[8]) {
  if (base + 8 <= n && ((reinterpret_cast<uintptr_t>(p + base) & 15u) == 0)) {
    if constexpr (LAST) {
      __stcs(reinterpret_cast<float4*>(p + base), make_float4(v[0], v[1], v[2], v[3]));
      __stcs(reinterpret_cast<float4*>(p + base) + 1, make_float4(v[4], v[5], v[6], v[7]));
    } else {
      Vec8<float>::store(p + base, v);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (base + i < n) p[base + i] = v[i];
  }
}

// sums[0] += <g + ef, g_hat>, sums[1] += <g_hat, g_hat>
// The CTAs' parts meet in 64 bits where the caller has room for that (Sum): a thousand of them added in FP32, in any order, moved the gain by 1e-7 to 1e-6.
template <typename T, typename Sum>
__global__ void __launch_bounds__(kThreads) packet_gain_kernel(const T* __restrict__ grad, const float* __restrict__ curr,
                                                               const float* __restrict__ prev, const float* __restrict__ ef,
                                                               float mu, int64_t n, Sum* __restrict__ sums) {
  float xp = 0.0f, pp = 0.0f;
  const int64_t stride = int64_t(gridDim.x) * kThreads * kPer;
  for (int64_t base = (int64_t(blockIdx.x) * kThreads + threadIdx.x) * kPer; base < n; base += stride) {
    float g[8], c[8], p[8], e[8];
    load8_any(grad, base, n, g);
    load8_f32(curr, base, n, c);
    load8_f32(prev, base, n, p);
    load8_f32(ef, base, n, e);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float pred = __fmaf_rn(mu, c[i] - p[i], c[i]);
      xp = __fmaf_rn(sanitize(g[i]) + e[i], pred, xp);
      pp = __fmaf_rn(pred, pred, pp);
    }
  }
  __shared__ float red[2][kThreads / 32];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    xp += __shfl_xor_sync(0xffffffffu, xp, off);
    pp += __shfl_xor_sync(0xffffffffu, pp, off);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = xp;
    red[1][threadIdx.x >> 5] = pp;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    Sum a = Sum(0);
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) a += Sum(red[threadIdx.x][i]);
    atomicAdd(&sums[threadIdx.x], a);
  }
}

// kappa: fixed (>= 0) or taken from the inner products in `sums` (fixed < 0). Thread 0 of block 0 writes the value
// it used into the payload's gain field.
template <typename Sum>
__device__ __forceinline__ float resolve_gain(float fixed, const Sum* sums) {
  if (fixed >= 0.0f) return fixed;
  const float xp = float(sums[0]), pp = float(sums[1]);
  return pp > 0.0f ? fminf(fmaxf(xp / pp, 0.0f), 1.0f) : 0.0f;
}

// The words in front of the gain that the host knows: a whole packet's header and its payload's fixed words, or none.
struct PacketHead {
  uint32_t word[12];
  uint32_t* dst;  // NULL: none
};

template <typename T, typename Sum>
__global__ void __launch_bounds__(kThreads) packet_encode_kernel(const T* __restrict__ grad, const float* __restrict__ curr,
                                                                 const float* __restrict__ prev, float* __restrict__ ef,
                                                                 float mu, float fixed_gain, const Sum* __restrict__ sums,
                                                                 int64_t n, float* __restrict__ gain_out,
                                                                 float* __restrict__ scales, uint8_t* __restrict__ packed,
                                                                 const __grid_constant__ PacketHead head) {
  const float kappa = resolve_gain(fixed_gain, sums);
  if (head.dst != nullptr && blockIdx.x == 0 && threadIdx.x < 12) head.dst[threadIdx.x] = head.word[threadIdx.x];
  if (blockIdx.x == 0 && threadIdx.x == 0) *gain_out = kappa;
  // whole tiles: every lane of a warp runs the same number of iterations (shuffles below)
  for (int64_t tile = tiles_of(n) - 1 - blockIdx.x; tile >= 0; tile -= gridDim.x) {
    const int64_t base = tile * kTile + threadIdx.x * kPer;
    float g[8], c[8], p[8], e[8];
    load8_any<true>(grad, base, n, g);
    load8_f32(curr, base, n, c);
    load8_f32(prev, base, n, p);
    load8_f32<true>(ef, base, n, e);
    float x[8], amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float pred = __fmaf_rn(mu, c[i] - p[i], c[i]);
      x[i] = sanitize(g[i]) + e[i] - kappa * pred;
      amax = fmaxf(amax, fabsf(x[i]));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    const float s = __fdiv_rn(amax, 7.0f);  // the host quantizer's scale, bit for bit
    uint32_t word = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float q = 0.0f;
      if (s > 0.0f) {
        const float scaled = __fdiv_rn(x[i], s);
        const float fl = floorf(scaled);
        q = (scaled - fl >= 0.5f) ? fl + 1.0f : fl;
        q = fminf(fmaxf(q, -8.0f), 7.0f);
      }
      x[i] -= q * s;  // what was not sent
      word |= (uint32_t(int(q)) & 0xFu) << (4 * i);
    }
    if (base < n) {
      if ((threadIdx.x & 7) == 0) scales[base / 64] = s;
      const int64_t byte0 = base / 2;
      const int64_t nbytes = (n + 1) / 2;
      if (byte0 + 4 <= nbytes && ((reinterpret_cast<uintptr_t>(packed + byte0) & 3u) == 0)) {
        *reinterpret_cast<uint32_t*>(packed + byte0) = word;
      } else {
        for (int k = 0; k < 4 && byte0 + k < nbytes; ++k) packed[byte0 + k] = uint8_t(word >> (8 * k));
      }
      if (ef != nullptr) store8_f32<true>(ef, base, n, x);
    }
  }
}

// What the words in front of a payload have to be for the decoder to run: of a launch that is queued before the host has seen the packet.
struct PacketExpect {
  const uint32_t* packet;  // NULL: the host has looked already
  uint32_t magic_version;  // low three bytes of the first word
  uint32_t flags_set, flags_clear;
  uint32_t layer, numel;
};
__device__ __forceinline__ bool as_expected(const PacketExpect& e) {
  if (e.packet == nullptr) return true;
  const uint32_t first = e.packet[0], flags = first >> 24;
  return (first & 0xffffffu) == e.magic_version && (flags & e.flags_set) == e.flags_set && (flags & e.flags_clear) == 0u && e.packet[2] == e.layer &&
         e.packet[8] == 0xc2800000u /* -64.0f */ && e.packet[9] == e.numel && e.packet[10] == 1u;
}

__global__ void __launch_bounds__(kThreads) packet_decode_kernel(const float* __restrict__ scales, const uint8_t* __restrict__ packed,
                                                                 const float* __restrict__ curr, const float* __restrict__ prev,
                                                                 float mu, float fixed_gain, const float* __restrict__ gain_in,
                                                                 int64_t n, float* __restrict__ out, const __grid_constant__ PacketExpect expect) {
  if (!as_expected(expect)) return;
  const float kappa = fixed_gain >= 0.0f ? fixed_gain : *gain_in;
  const int64_t nbytes = (n + 1) / 2;
  const int64_t stride = int64_t(gridDim.x) * kTile;
  for (int64_t base = (int64_t(blockIdx.x) * kThreads + threadIdx.x) * kPer; base < n; base += stride) {
    const int64_t byte0 = base / 2;
    uint32_t word = 0u;
    if (byte0 + 4 <= nbytes && ((reinterpret_cast<uintptr_t>(packed + byte0) & 3u) == 0)) {
      word = *reinterpret_cast<const uint32_t*>(packed + byte0);
    } else {
      for (int k = 0; k < 4 && byte0 + k < nbytes; ++k) word |= uint32_t(packed[byte0 + k]) << (8 * k);
    }
    const float s = scales[base / 64];
    float c[8], p[8];
    load8_f32<true>(kappa != 0.0f ? curr : nullptr, base, n, c);
    load8_f32<true>(kappa != 0.0f ? prev : nullptr, base, n, p);
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = int(word << (28 - 4 * i)) >> 28;
      o[i] = __fmaf_rn(kappa, __fmaf_rn(mu, c[i] - p[i], c[i]), float(q) * s);
    }
    store8_f32(out, base, n, o);
  }
}

// The words that the host wants to see, into memory of the host's that the device can write: two copies of a few bytes take three
// times as long. (One warp; the checksum is read after everything before this launch is complete.)
__global__ void packet_report_kernel(const uint8_t* __restrict__ packet, int bytes, const uint32_t* __restrict__ crc, uint8_t* __restrict__ host) {
  for (int i = threadIdx.x; i < bytes; i += 32) host[i] = packet[i];
  if (threadIdx.x == 0 && crc != nullptr) *reinterpret_cast<uint32_t*>(host + 44) = *crc;
}

// The encoder and the decoder: four tiles a CTA (the first of them waits for the gain), which the hardware hands out as SMs come free, but not
// fewer CTAs than fill the device. (The gains keep a grid of fixed size: how their sums are grouped decides their rounding.)
int tiles_grid(int64_t n) { return int(std::min<int64_t>(tiles_of(n), std::max<int64_t>(kMaxBlocks, (tiles_of(n) + 3) / 4))); }

int grid_for(int64_t n) {
  const int64_t blocks = (n + int64_t(kThreads) * kPer - 1) / (int64_t(kThreads) * kPer);
  return int(blocks < 1 ? 1 : blocks > kMaxBlocks ? kMaxBlocks : blocks);
}

}  // namespace
}  // namespace nangila

extern "C" int64_t nangila_packet_payload_bytes(int64_t n) { return 20 + 4 * ((n + 63) / 64) + (n + 1) / 2; }

namespace nangila {
namespace {
// `sums`: two numbers for the inner products, used when the gain is to be derived.
template <typename Sum>
cudaError_t launch_encode(const void* grad, int32_t dtype, const float* curr, const float* prev, float* ef, float mu, float gain, int64_t n,
                          uint8_t* payload, Sum* sums, const PacketHead& head, cudaStream_t stream) {
  float* gain_out = reinterpret_cast<float*>(payload + 16);
  float* scales = reinterpret_cast<float*>(payload + 20);
  uint8_t* packed = payload + 20 + 4 * ((n + 63) / 64);
  const int grid = grid_for(n);
  if (curr == nullptr) gain = 0.0f;
  if (gain < 0.0f) {
    const cudaError_t e = cudaMemsetAsync(sums, 0, 2 * sizeof(Sum), stream);
    if (e != cudaSuccess) return e;
  }
#define NANGILA_PACKET_LAUNCH(TYPE)                                                                                  \
  do {                                                                                                               \
    if (gain < 0.0f)                                                                                                 \
      packet_gain_kernel<TYPE, Sum><<<grid, kThreads, 0, stream>>>(static_cast<const TYPE*>(grad), curr, prev, ef, mu, n, sums); \
    packet_encode_kernel<TYPE, Sum><<<tiles_grid(n), kThreads, 0, stream>>>(static_cast<const TYPE*>(grad), curr, prev, ef, mu, gain, \
                                                              sums, n, gain_out, scales, packed, head);              \
  } while (0)
  switch (dtype) {
    case NANGILA_F32: NANGILA_PACKET_LAUNCH(float); break;
    case NANGILA_BF16: NANGILA_PACKET_LAUNCH(__nv_bfloat16); break;
    case NANGILA_F16: NANGILA_PACKET_LAUNCH(__half); break;
    default: return cudaErrorInvalidValue;
  }
#undef NANGILA_PACKET_LAUNCH
  return cudaGetLastError();
}

// fixed words of the payload: block size (negated), numel, ndim, dim
void fixed_words(int64_t n, uint32_t* w) {
  const float neg_block = -64.0f;
  memcpy(&w[0], &neg_block, 4);
  w[1] = w[3] = uint32_t(n);
  w[2] = 1u;
}

bool bad_encode(const void* grad, const float* curr, const float* prev, float mu, int64_t n, const uint8_t* out) {
  return grad == nullptr || out == nullptr || n <= 0 || n > 0x7fffffffll || (reinterpret_cast<uintptr_t>(out) & 3u) != 0 ||
         (curr == nullptr) != (prev == nullptr) || !(mu >= 0.0f && mu <= 1.0f);
}

}  // namespace
}  // namespace nangila

extern "C" int nangila_packet_encode(const void* grad, int32_t dtype, const float* curr, const float* prev, float* ef, float mu,
                                     float gain, int64_t n, uint8_t* payload, cudaStream_t stream) {
  using namespace nangila;
  if (bad_encode(grad, curr, prev, mu, n, payload)) return int(cudaErrorInvalidValue);
  // The two inner products live in the first 8 bytes of the payload until the encoder has read them; the
  // fixed words that belong there are copied in afterwards (the encoder never writes the first 16 bytes).
  const PacketHead head{};
  const cudaError_t e = launch_encode(grad, dtype, curr, prev, ef, mu, gain, n, payload, reinterpret_cast<float*>(payload), head, stream);
  if (e != cudaSuccess) return int(e);
  uint32_t words[4];
  fixed_words(n, words);
  // pageable source: the runtime stages it before the call returns, so the stack buffer may go away
  return int(cudaMemcpyAsync(payload, words, 16, cudaMemcpyHostToDevice, stream));
}

// A whole packet, header and checksum included, in two or three launches and no copy: the encoder writes the words that the host
// knows from its own parameters, and the checksum kernel puts its result where it belongs. For small layers the call is what
// costs: 10 007 FP32 elements through compress_gpu, decompress_gpu and update_gpu took 142 us with the header and the checksum copied in by
// tensor operations and two synchronisations before decoding, 91 us this way.
namespace nangila {
namespace {
template <typename Sum>
int compress(const void* grad, int32_t dtype, const float* curr, const float* prev, float* ef, float mu, float gain, int64_t n, const uint8_t* header,
             uint8_t* packet, Sum* sums, cudaStream_t stream) {
  if (bad_encode(grad, curr, prev, mu, n, packet) || header == nullptr || sums == nullptr) return int(cudaErrorInvalidValue);
  PacketHead head;
  memcpy(head.word, header, 32);
  head.word[3] = 0u;  // the checksum's place
  fixed_words(n, head.word + 8);
  head.dst = reinterpret_cast<uint32_t*>(packet);
  const cudaError_t e = launch_encode(grad, dtype, curr, prev, ef, mu, gain, n, packet + 32, sums, head, stream);
  if (e != cudaSuccess) return int(e);
  uint32_t* crc = reinterpret_cast<uint32_t*>(packet + 12);
  return nangila_crc32_cleared(packet + 32, nangila_packet_payload_bytes(n), crc, stream);  // the encoder has written the header
}
}  // namespace
}  // namespace nangila

extern "C" int nangila_packet_compress(const void* grad, int32_t dtype, const float* curr, const float* prev, float* ef, float mu,
                                       float gain, int64_t n, const uint8_t* header, uint8_t* packet, float* sums, cudaStream_t stream) {
  return nangila::compress(grad, dtype, curr, prev, ef, mu, gain, n, header, packet, sums, stream);
}
extern "C" int nangila_packet_compress_f64(const void* grad, int32_t dtype, const float* curr, const float* prev, float* ef, float mu,
                                           float gain, int64_t n, const uint8_t* header, uint8_t* packet, double* sums, cudaStream_t stream) {
  return nangila::compress(grad, dtype, curr, prev, ef, mu, gain, n, header, packet, sums, stream);
}

namespace nangila {
namespace {
int launch_decode(const uint8_t* payload, int64_t payload_bytes, int32_t ndim, const float* curr, const float* prev, float mu, float gain, int64_t n,
                  float* out, const PacketExpect& expect, cudaStream_t stream) {
  if (payload == nullptr || out == nullptr || n <= 0 || ndim < 0 || ndim > 8 || (reinterpret_cast<uintptr_t>(payload) & 3u) != 0 ||
      (curr == nullptr) != (prev == nullptr))
    return int(cudaErrorInvalidValue);
  const int64_t off_gain = 12 + 4 * int64_t(ndim);
  const int64_t need = off_gain + 4 + 4 * ((n + 63) / 64) + (n + 1) / 2;
  if (payload_bytes < need) return int(cudaErrorInvalidValue);
  const float* gain_in = reinterpret_cast<const float*>(payload + off_gain);
  const float* scales = gain_in + 1;
  const uint8_t* packed = reinterpret_cast<const uint8_t*>(scales + (n + 63) / 64);
  if (curr == nullptr) gain = 0.0f;
  packet_decode_kernel<<<tiles_grid(n), kThreads, 0, stream>>>(scales, packed, curr, prev, mu, gain, gain_in, n, out, expect);
  return int(cudaGetLastError());
}
}  // namespace
}  // namespace nangila

extern "C" int nangila_packet_decode(const uint8_t* payload, int64_t payload_bytes, int32_t ndim, const float* curr,
                                     const float* prev, float mu, float gain, int64_t n, float* out, cudaStream_t stream) {
  return nangila::launch_decode(payload, payload_bytes, ndim, curr, prev, mu, gain, n, out, nangila::PacketExpect{}, stream);
}

// Queues the decoder for a packet whose header the host has not seen yet. It runs if the packet is what the receiver of layer `layer` expects (a
// driver's one-dimensional packet of n elements in blocks of 64, with a prediction exactly if curr is given) and leaves `out` as it is
// otherwise. cudaErrorInvalidValue if the packet is too short for that.
extern "C" int nangila_packet_decode_expected(const uint8_t* packet, int64_t packet_bytes, uint32_t layer, const float* curr, const float* prev, float mu,
                                              int64_t n, float* out, cudaStream_t stream) {
  using namespace nangila;
  if (packet == nullptr || packet_bytes <= 32 || n > 0xffffffffll) return int(cudaErrorInvalidValue);
  const PacketExpect e{reinterpret_cast<const uint32_t*>(packet), 0x014e47u, 0x02u, curr != nullptr ? 0x80u : 0u, layer, uint32_t(n)};
  return launch_decode(packet + 32, packet_bytes - 32, 1, curr, prev, mu, curr != nullptr ? -1.0f : 0.0f, n, out, e, stream);
}

// `host`: 48 bytes of pinned memory; gets the first `bytes` (at most 44) of the packet and, at byte 44, *crc.
extern "C" int nangila_packet_report(const uint8_t* packet, int32_t bytes, const uint32_t* crc, uint8_t* host, cudaStream_t stream) {
  using namespace nangila;
  if (packet == nullptr || host == nullptr || bytes < 0 || bytes > 44 || (reinterpret_cast<uintptr_t>(host) & 3u) != 0) return int(cudaErrorInvalidValue);
  packet_report_kernel<<<1, 32, 0, stream>>>(packet, bytes, crc, host);
  return int(cudaGetLastError());
}

// Small runtime helpers for callers that bind this library without linking the CUDA runtime themselves
// (the host core's C entry points).
extern "C" int nangila_copy_to_host(void* dst, const void* src, int64_t nbytes, cudaStream_t stream) {
  cudaError_t e = cudaMemcpyAsync(dst, src, size_t(nbytes), cudaMemcpyDeviceToHost, stream);
  if (e != cudaSuccess) return int(e);
  return int(cudaStreamSynchronize(stream));
}
extern "C" int nangila_copy_to_device(void* dst, const void* src, int64_t nbytes, cudaStream_t stream) {
  return int(cudaMemcpyAsync(dst, src, size_t(nbytes), cudaMemcpyHostToDevice, stream));
}
extern "C" int nangila_stream_sync(cudaStream_t stream) { return int(cudaStreamSynchronize(stream)); }
