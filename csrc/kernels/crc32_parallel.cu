// Parallel IEEE CRC32 (polynomial 0xEDB88320, initial value and final XOR 0xFFFFFFFF) of a device buffer.
//
// The CRC register is linear over GF(2): with w_i the 32-bit words of the message and polynomials taken mod P,
//   crc = sum_i w_i x^(32 + 8 bytes behind word i)  +  0xFFFFFFFF x^(8 nbytes)  +  0xFFFFFFFF.
// Every thread runs Horner's rule over the 16-byte groups g, g + G, g + 2 G, ... (G = threads of the grid): its four words
// are four independent states that are multiplied by the one constant x^(128 G) per step. Neighbouring threads read
// neighbouring groups, so loads are whole lines; the groups are counted from the END of the message, so that every thread
// ends G - 1 - g groups before it and the missing groups are leading zeros, which leave a zero state as it is. At the end
// each state is multiplied by its distance to the end and everything is added up with XOR, in any order.
//
// What bounds it: the multiplication by x^(128 G) is seven table look-ups in shared memory, one per five bits: 32 entries are
// 32 banks, so the look-ups of a warp never collide (nibbles need eight; byte tables need four, but the random bytes of 32
// lanes meet 3-4 deep in a bank). With about 25 instructions per word the issue rate and the look-ups cost about as much as
// each other. Measured on B200: a 21.7 MB packet 1.40 ms -> 14.4 us, a 6 KB one 88 -> 5.4 us; before, each thread walked 512 bytes of its
// own with a byte table and one block combined the 42 000 partial sums in 16 rounds, squaring its way to every power.
//
// Replaces compute_crc32_kernel (nangila-cuda/src/kernels/crc32.cu:56-72), which walks the whole
// payload with a single thread, and matches the host table CRC (nangila-core/src/packet.rs:241-274).
#include <cuda_runtime.h>

#include "nangila_kernels.h"
#include "nangila_noalloc.h"

namespace nangila {
namespace {

constexpr uint32_t kPoly = 0xEDB88320u;
constexpr uint32_t kOne = 0x80000000u;  // x^0 in the reflected bit order (bit 31 is x^0)
constexpr int kThreads = 256;
// One CTA does the whole buffer up to eight steps per thread (32 KB): it stores the result itself, where several CTAs
// need the word cleared first, and the launch that saves costs about as much as those steps.
constexpr int64_t kOneCtaSteps = 8;
constexpr int kMaxCtas = 592;  // four per SM

// a * b mod P; constant trip count, so that independent products overlap.
__host__ __device__ constexpr uint32_t mulmod(uint32_t a, uint32_t b) {
  uint32_t p = 0;
  for (int i = 31; i >= 0; --i) {
    p ^= b & (0u - ((a >> i) & 1u));
    b = (b >> 1) ^ (kPoly & (0u - (b & 1u)));
  }
  return p;
}
constexpr uint32_t mul_x(uint32_t a, int n) {  // a * x^n
  for (int i = 0; i < n; ++i) a = (a >> 1) ^ (kPoly & (0u - (a & 1u)));
  return a;
}

// Multiplication by a constant c, five bits at a time: table[32 t + v] = (v << 5 t) c.
constexpr int kPieces = 7, kEntries = kPieces * 32;
__device__ __forceinline__ uint32_t times(const uint32_t* table, uint32_t x) {
  const char* t = reinterpret_cast<const char*>(table);
  uint32_t r = *reinterpret_cast<const uint32_t*>(t + ((x << 2) & 0x7cu));
#pragma unroll
  for (int k = 1; k < kPieces; ++k) r ^= *reinterpret_cast<const uint32_t*>(t + k * 128 + ((x >> (5 * k - 2)) & 0x7cu));
  return r;
}
static_assert(kEntries <= kThreads, "one thread per entry");

// Constants of the last part, made by the compiler: the table of x^32, and x^(128 d), x^(128 32 d), x^(128 256 d), x^(128 256 16 d),
// x^(128 256 256 d): the factors of d groups, warps, CTAs, 16 CTAs, 256 CTAs.
struct Constants {
  uint32_t word[kEntries];
  uint32_t lane[32], warp[8], cta[3][16];
};
constexpr Constants make_constants() {
  Constants c{};
  constexpr uint32_t x32 = mul_x(kOne, 32);
  for (int e = 0; e < kEntries; ++e) c.word[e] = mulmod(uint32_t(e & 31) << (5 * (e >> 5)), x32);
  uint32_t step = mul_x(kOne, 128);
  c.lane[0] = c.warp[0] = kOne;
  for (int d = 1; d < 32; ++d) c.lane[d] = mulmod(c.lane[d - 1], step);
  step = mulmod(c.lane[31], step);
  for (int d = 1; d < 8; ++d) c.warp[d] = mulmod(c.warp[d - 1], step);
  step = mulmod(c.warp[7], step);
  for (int k = 0; k < 3; ++k) {
    c.cta[k][0] = kOne;
    for (int d = 1; d < 16; ++d) c.cta[k][d] = mulmod(c.cta[k][d - 1], step);
    step = mulmod(c.cta[k][15], step);
  }
  return c;
}
__constant__ Constants c_crc = make_constants();
static_assert(kThreads == 256 && kMaxCtas < 16 * 16 * 16, "the constants above");

struct CrcArgs {
  const uint8_t* data;   // first byte of the message
  int64_t head;          // bytes before the first 16-byte boundary of memory
  int64_t groups;        // whole 16-byte groups after them
  int32_t tail;          // bytes after those
  uint32_t step;         // x^(128 G)
  uint32_t head_factor;  // x^(8 (nbytes - head))
  uint32_t tail_factor;  // x^(8 tail)
  uint32_t fixed;        // 0xFFFFFFFF x^(8 nbytes) + 0xFFFFFFFF
  uint32_t* out;
};

// CRC register after `n` bytes, starting from 0.
__device__ __forceinline__ uint32_t crc_bytes(const uint8_t* p, int n) {
  uint32_t c = 0;
  for (int i = 0; i < n; ++i) {
    c ^= p[i];
#pragma unroll
    for (int k = 0; k < 8; ++k) c = (c >> 1) ^ (kPoly & (0u - (c & 1u)));
  }
  return c;
}

__global__ void __launch_bounds__(kThreads) crc_kernel(const __grid_constant__ CrcArgs a) {
  __shared__ uint32_t by_step[kEntries], by_word[kEntries];
  __shared__ uint32_t part[kThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t G = int64_t(gridDim.x) * kThreads, g = int64_t(blockIdx.x) * kThreads + tid;
  const int steps = int((a.groups + G - 1) / G);
  const uint4* p = reinterpret_cast<const uint4*>(a.data + a.head);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  int64_t q = g - (steps * G - a.groups);  // counted from the end: negative in the first step of the leading threads
  uint4 w0 = q >= 0 && steps > 0 ? __ldg(p + q) : zero;
  uint4 w1 = steps > 1 ? __ldg(p + q + G) : zero;
  if (tid < kEntries) {
    by_step[tid] = steps > 1 ? mulmod(uint32_t(tid & 31) << (5 * (tid >> 5)), a.step) : 0u;
    by_word[tid] = c_crc.word[tid];
  }
  __syncthreads();
  uint32_t s[4] = {w0.x, w0.y, w0.z, w0.w};
  for (int k = 1; k < steps; ++k) {
    q += G;
    const uint4 w2 = k + 1 < steps ? __ldg(p + q + G) : zero;
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = times(by_step, s[j]);
    s[0] ^= w1.x; s[1] ^= w1.y; s[2] ^= w1.z; s[3] ^= w1.w;
    w1 = w2;
  }
  uint32_t v = times(by_word, s[0]) ^ s[1];
  v = times(by_word, v) ^ s[2];
  v = times(by_word, v) ^ s[3];
  v = __reduce_xor_sync(0xffffffffu, mulmod(times(by_word, v), c_crc.lane[31 - lane]));
  if (lane == 0) part[tid >> 5] = v;
  __syncthreads();
  if (tid >= 32) return;
  v = lane < kThreads / 32 ? mulmod(part[lane], c_crc.warp[kThreads / 32 - 1 - lane]) : 0u;
  v = __reduce_xor_sync(0xffffffffu, v);
  if (lane == 0) {
    const uint32_t b = gridDim.x - 1 - blockIdx.x;  // CTAs behind this one
    const uint32_t behind = mulmod(mulmod(c_crc.cta[0][b & 15], c_crc.cta[1][(b >> 4) & 15]), c_crc.cta[2][b >> 8]);
    v = mulmod(behind, mulmod(v, a.tail_factor));
    if (blockIdx.x == 0) {
      v ^= a.fixed;
      if (a.head > 0) v ^= mulmod(crc_bytes(a.data, int(a.head)), a.head_factor);
      if (a.tail > 0) v ^= crc_bytes(a.data + a.head + a.groups * 16, a.tail);
    }
    if (gridDim.x == 1) *a.out = v;
    else atomicXor(a.out, v);  // *out was cleared before the launch
  }
}

// x^(8 n)
uint32_t x_pow_bytes(uint64_t n) {
  struct Squares {
    uint32_t v[64];
    Squares() {
      v[0] = mul_x(kOne, 8);
      for (int i = 1; i < 64; ++i) v[i] = mulmod(v[i - 1], v[i - 1]);
    }
  };
  static const Squares squares;
  uint32_t r = kOne;
  for (int i = 0; n != 0; ++i, n >>= 1)
    if (n & 1u) r = mulmod(r, squares.v[i]);
  return r;
}

// cleared: *out is zero when the kernel starts.
cudaError_t launch_crc(const void* data, int64_t nbytes, uint32_t* out, bool cleared, cudaStream_t stream) {
  CrcArgs a;
  a.data = static_cast<const uint8_t*>(data);
  a.head = int64_t((16u - (reinterpret_cast<uintptr_t>(data) & 15u)) & 15u);
  if (a.head > nbytes) a.head = nbytes;
  a.groups = (nbytes - a.head) / 16;
  a.tail = int32_t((nbytes - a.head) % 16);
  int64_t ctas = 1;
  if (a.groups > kOneCtaSteps * kThreads) {
    ctas = (a.groups + 4 * kThreads - 1) / (4 * kThreads);  // at least four steps per thread
    if (ctas > kMaxCtas) ctas = kMaxCtas;
  }
  a.step = x_pow_bytes(uint64_t(ctas) * kThreads * 16);
  a.head_factor = x_pow_bytes(uint64_t(nbytes - a.head));
  a.tail_factor = x_pow_bytes(uint64_t(a.tail));
  a.fixed = mulmod(0xFFFFFFFFu, x_pow_bytes(uint64_t(nbytes))) ^ 0xFFFFFFFFu;
  a.out = out;
  if (ctas > 1 && !cleared) {
    const cudaError_t e = cudaMemsetAsync(out, 0, 4, stream);
    if (e != cudaSuccess) return e;
  }
  crc_kernel<<<unsigned(ctas), kThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace
}  // namespace nangila

// The kernel keeps nothing in memory; the word is what callers that allocate a table get to allocate.
extern "C" int64_t nangila_crc32_scratch_words(int64_t) { return 1; }

// out: one uint32 on the device. `scratch` is not used (it was a table of partial sums); as before it may be NULL only for
// an empty buffer.
extern "C" int nangila_crc32(const void* data, int64_t nbytes, uint32_t* scratch, uint32_t* out, cudaStream_t stream) {
  if (out == nullptr || nbytes < 0 || (nbytes > 0 && (data == nullptr || scratch == nullptr)))
    return int(cudaErrorInvalidValue);
  if (nbytes == 0) return int(cudaMemsetAsync(out, 0, 4, stream));
  return int(nangila::launch_crc(data, nbytes, out, false, stream));
}

// The same with *out known to be zero: one launch instead of a memset and a launch where several CTAs add to it.
extern "C" int nangila_crc32_cleared(const void* data, int64_t nbytes, uint32_t* out, cudaStream_t stream) {
  if (out == nullptr || nbytes <= 0 || data == nullptr) return int(cudaErrorInvalidValue);
  return int(nangila::launch_crc(data, nbytes, out, true, stream));
}

// Allocation-free entry point (declared in nangila_noalloc.h; the reference has nothing like it).
extern "C" int64_t nangila_crc32_noalloc_max_bytes(void) { return int64_t(64) << 20; }

extern "C" int nangila_crc32_noalloc(const void* data, int64_t nbytes, uint32_t* out, cudaStream_t stream) {
  if (out == nullptr || nbytes < 0 || (nbytes > 0 && data == nullptr)) return int(cudaErrorInvalidValue);
  if (nbytes > nangila_crc32_noalloc_max_bytes()) return int(cudaErrorInvalidValue);
  if (nbytes == 0) return int(cudaMemsetAsync(out, 0, 4, stream));
  return int(nangila::launch_crc(data, nbytes, out, false, stream));
}
