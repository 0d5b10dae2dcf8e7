// PowerSGD on Blackwell tensor cores (sm_100a).
//
// For one gradient matrix M (m x n, row-major; M = gradient + error memory, bf16) and rank r <= 16:
//   prep         M <- bf16(grad + error memory)
//   GEMM A       P_local  = M  * Q        (m x 16)   tcgen05.mma, A = M  tiles (K-major),  B = Q^T (16 x n)
//   exchange     P = mean over ranks of P_local; Gram-Schmidt on the columns of P (in-kernel)
//   GEMM B       Q'_local = M^T * P       (n x 16)   tcgen05.mma, A = M^T tiles (MN-major), B = P^T (16 x m)
//   exchange     Q' = mean over ranks of Q'_local; orthonormalised copy kept as the next warm start
//   reconstruct  grad <- P Q'^T ; error memory <- M - P Q'^T
// Both GEMMs run as 128 x 16 output tiles: operands are staged in shared memory by TMA
// (cp.async.bulk.tensor, 128-byte swizzle, no cluster multicast) through a 4-stage mbarrier pipeline,
// one elected thread issues tcgen05.mma with the accumulator in tensor memory, and the epilogue reads
// it back with tcgen05.ld. M is read straight from its row-major storage in both GEMMs: the second
// one feeds the tensor core an MN-major A operand instead of materialising a transpose.
// The exchanges store each rank's factor into every rank's slot over NVLink and every rank then adds
// the W slots in rank order, so all replicas hold bit-identical P and Q'.
//
// What it replaces in the reference: PowerSGDCompressor::compress / decompress
// (nangila-core/src/power_sgd.rs:46-193: ndarray GEMMs on the host, per-rank factors shipped and W
// dense reconstructions averaged). Here P and Q' are averaged across ranks (standard PowerSGD).
#include <algorithm>
#include <cstring>
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "follow.cuh"
#include "nangila_kernels.h"
#include "ptx_sm100.cuh"
#include "quant.cuh"
#include "signal.cuh"
#include "warp_sums.cuh"

namespace nangila {
namespace {
namespace cg = cooperative_groups;

using namespace sm100;
using namespace comm;

constexpr int kTileRows = 128;   // UMMA M
constexpr int kCols = 16;        // UMMA N: rank padded to 16
constexpr int kSlabK = 64;       // bf16 elements per 128-byte swizzle row
constexpr int kStages = 4;
constexpr int kABytes = kTileRows * kSlabK * 2;  // 16 KiB
constexpr int kBBytes = kCols * kSlabK * 2;      // 2 KiB
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kGemmThreads = 128;
constexpr int kTmemCols = 32;
constexpr int kGemmSmem = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers and flags*/;

// One CTA computes out[row0 .. row0+127][0..15] (+)= sum over its K range.
//  A_MN = false: tmA is a map of M (inner dim = K), box {64, 128}; the A stage is one box.
//  A_MN = true : tmA is a map of M whose inner dim is the OUTPUT row dimension, box {64, 64}; the A
//                stage is two boxes (output rows 0..63 and 64..127) of 64 K-rows each.
//  tmB always maps B^T (16 x K, inner dim = K), box {64, 16}.
template <bool A_MN>
__global__ void __launch_bounds__(kGemmThreads)
psgd_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 float* __restrict__ out, int rows_out, int k_total, int k_per_split, int use_atomics, int columns,
                 uint32_t* status, uint64_t timeout_ns, const __grid_constant__ NangilaPsgdPush push) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* accum_done = empty + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum_done + 1);
  uint32_t* failed = tmem_slot + 1;
  uint32_t* last_of_tile = failed + 1;   // this CTA completed its row tile (epilogue push)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * kTileRows;
  const int k_begin = blockIdx.y * k_per_split;
  const int k_end = min(k_total, k_begin + k_per_split);
  const int nslabs = (k_end - k_begin + kSlabK - 1) / kSlabK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accum_done, 1);
    *failed = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
  }
  if (warp == 0) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (push.counters == nullptr) may_follow();
  follow();

  if (nslabs > 0) {
    if (warp == 0 && lane == 0) {
      // ---------------- TMA producer ----------------
      for (int i = 0; i < nslabs; ++i) {
        const int s = i % kStages;
        if (i >= kStages && !mbar_wait(&empty[s], uint32_t((i / kStages - 1) & 1), timeout_ns)) {
          *failed = 1;
          break;
        }
        uint8_t* a_dst = smem + s * kStageBytes;
        uint8_t* b_dst = a_dst + kABytes;
        const int k0 = k_begin + i * kSlabK;
        mbar_arrive_expect_tx(&full[s], kStageBytes);
        if (A_MN) {
          tma_load_2d(a_dst, &tmA, row0, k0, &full[s]);
          tma_load_2d(a_dst + kABytes / 2, &tmA, row0 + 64, k0, &full[s]);
        } else {
          tma_load_2d(a_dst, &tmA, k0, row0, &full[s]);
        }
        tma_load_2d(b_dst, &tmB, k0, 0, &full[s]);
      }
    } else if (warp == 1 && lane == 0) {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc = make_idesc_bf16(kTileRows, kCols, A_MN, false);
      bool ok = true;
      for (int i = 0; i < nslabs && ok; ++i) {
        const int s = i % kStages;
        if (!mbar_wait(&full[s], uint32_t((i / kStages) & 1), timeout_ns)) {
          *failed = 1;
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t a_addr = smem_u32(smem + s * kStageBytes);
        const uint32_t b_addr = a_addr + kABytes;
#pragma unroll
        for (int kk = 0; kk < kSlabK / 16; ++kk) {
          // K-major: 16 elements along K = 32 bytes inside the swizzle row.
          // MN-major: 16 K-rows = two groups of 8 rows of 128 bytes.
          const uint64_t a_desc = A_MN ? make_smem_desc(a_addr + kk * 2048, kABytes / 2, 1024)
                                       : make_smem_desc(a_addr + kk * 32, 16, 1024);
          const uint64_t b_desc = make_smem_desc(b_addr + kk * 32, 16, 1024);
          umma_bf16(tmem_base, a_desc, b_desc, idesc, (i > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(&empty[s]);  // frees the stage once these MMAs have read it
      }
      if (ok) umma_commit(accum_done);
    }
    __syncwarp();
    // ---------------- epilogue: all four warps ----------------
    bool ok = mbar_wait(accum_done, 0, timeout_ns);
    if (*reinterpret_cast<volatile uint32_t*>(failed) != 0u) ok = false;
    ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld needs the whole warp
    if (ok) {
      tc_fence_after_sync();
      float v[16];
      tmem_ld_32x32b_x16(tmem_base + (uint32_t(warp * 32) << 16), v);
      const int row = row0 + warp * 32 + lane;
      if (row < rows_out) {
        float* dst = out + int64_t(row) * kCols;
        if (use_atomics) {
          // four columns per reduction, and none that nobody reads
#pragma unroll
          for (int c = 0; c < kCols; c += 4)
            if (c < columns)
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + c), "f"(v[c]), "f"(v[c + 1]), "f"(v[c + 2]), "f"(v[c + 3])
                           : "memory");
        } else {
#pragma unroll
          for (int c = 0; c < kCols; c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        }
      }
    } else if (threadIdx.x == 0) {
      report_failure(status, kTimeoutGrid, 0u, 0xffffffffu, 0u, 0u, 7u, uint32_t(blockIdx.x));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, kTmemCols);

  // ---------------- exchange started from the epilogue ----------------
  // Whichever of a tile's K splits arrives last finds the complete tile in `out` (its own part went there above,
  // the others' were fenced before they counted themselves in) and stores it into every rank's slot for this
  // rank. A CTA whose pipeline failed still counts itself in, so that nobody waits for it; the status block says
  // that the data is not to be trusted.
  if (push.counters != nullptr) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) *last_of_tile = atomicAdd(&push.counters[blockIdx.x], 1u) == gridDim.y - 1 ? 1u : 0u;
    __syncthreads();
    if (*last_of_tile != 0u) {
      __threadfence();
      const uint32_t epoch = push.epoch_dev != nullptr ? *push.epoch_dev : push.epoch;
      const int W = push.world, r = push.rank;
      const uint64_t slot_bytes = (uint64_t(rows_out) * r * 4 + 255) & ~uint64_t(255);
      const uint64_t base = push.recv_off + uint64_t(epoch & 1u) * W * slot_bytes + uint64_t(push.me) * slot_bytes;
      const int row = row0 + warp * 32 + lane;
      if (row < rows_out) {
        float v[kCols];
#pragma unroll
        for (int c = 0; c < kCols; c += 4) {
          if (c < r) {
            const float4 a = __ldcg(reinterpret_cast<const float4*>(out + int64_t(row) * kCols + c));
            v[c] = a.x; v[c + 1] = a.y; v[c + 2] = a.z; v[c + 3] = a.w;
          }
        }
        for (int d = 0; d < W; ++d) {
          float* dst = reinterpret_cast<float*>(push.region[(push.me + d) % W] + base);
#pragma unroll
          for (int c = 0; c < kCols; ++c)
            if (c < r) dst[int64_t(c) * rows_out + row] = v[c];   // adjacent rows: adjacent addresses
        }
      }
      if (W > 1) __threadfence_system();
      else __threadfence();  // nobody outside this GPU reads it
      __syncthreads();
      if (threadIdx.x == 0) {
        const uint32_t tiles = gridDim.x;
        if (atomicAdd(&push.counters[tiles], 1u) == tiles - 1) {
          if (W > 1) __threadfence_system();  // every tile's stores were fenced before its CTA counted itself in
          else __threadfence();
          for (int d = 0; d < W; ++d)
            st_release_sys(reinterpret_cast<uint32_t*>(push.region[d] + push.flag_off) + push.me, epoch);
        }
      }
    }
  }
}

// ---- prep / reconstruct (element-wise) -----------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) psgd_prep_kernel(const T* __restrict__ grad, const __nv_bfloat16* __restrict__ ef,
                                                       __nv_bfloat16* __restrict__ mef, int64_t numel,
                                                       float* __restrict__ z0, int64_t n0, float* __restrict__ z1,
                                                       int64_t n1) {
  may_follow();
  const int64_t t0 = int64_t(blockIdx.x) * 256 + threadIdx.x, stride = int64_t(gridDim.x) * 256;
  // Eight elements a thread where the addresses allow it (bound by HBM; one element a thread was bound by latency: 2.4 M elements
  // 4.7 -> 3.6 us).
  const bool vec = ((reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(ef) | reinterpret_cast<uintptr_t>(mef)) & 15u) == 0;
  const int64_t n8 = vec ? numel / 8 : 0;
  for (int64_t q = t0; q < n8; q += stride) {
    float g[8], e[8];
    dev::Vec8<T>::load(grad + q * 8, g);
    dev::Vec8<__nv_bfloat16>::load(ef + q * 8, e);
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] += dev::sanitize(g[k]);
    dev::Vec8<__nv_bfloat16>::store(mef + q * 8, e);
  }
  for (int64_t i = n8 * 8 + t0; i < numel; i += stride)
    mef[i] = __float2bfloat16_rn(dev::sanitize(dev::Vec16<T>::to_float(grad[i])) + __bfloat162float(ef[i]));
  // the two projections accumulate into these with atomics (split K): clear them here, not in launches of their own
  for (int64_t i = t0; i < n0; i += stride) z0[i] = 0.0f;
  for (int64_t i = t0; i < n1; i += stride) z1[i] = 0.0f;
}
// grad = P Q^T (rank r), ef = (m + ef) - grad. P and Q are the averaged factors, COLUMN-major
// (P[k * m + row], Q[k * n + col]). Each thread owns 8 consecutive columns and walks down the rows of
// its CTA's share; for r <= 4 its 8 x r slice of Q stays in registers, so per row it reads 16 bytes of
// m + ef and r broadcast values of P and writes the 8 results twice (bucket, error memory).
template <typename T, int RQ>
__global__ void __launch_bounds__(256) psgd_reconstruct_kernel(T* __restrict__ grad, __nv_bfloat16* __restrict__ ef,
                                                              const __nv_bfloat16* __restrict__ mef,
                                                              const float* __restrict__ P, const float* __restrict__ Q,
                                                              int m, int n, int r) {
  follow();
  const int col = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (col >= n) return;  // n is a multiple of 8
  float q[RQ > 0 ? RQ : 1][8];
  if constexpr (RQ > 0) {
#pragma unroll
    for (int k = 0; k < RQ; ++k) {
      if (k < r) dev::Vec8<float>::load(Q + int64_t(k) * n + col, q[k]);
      else {
#pragma unroll
        for (int j = 0; j < 8; ++j) q[k][j] = 0.0f;
      }
    }
  }
  for (int row = blockIdx.y; row < m; row += gridDim.y) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
    if constexpr (RQ > 0) {
#pragma unroll
      for (int k = 0; k < RQ; ++k) {
        const float pk = k < r ? P[int64_t(k) * m + row] : 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = __fmaf_rn(pk, q[k][j], acc[j]);
      }
    } else {
      for (int k = 0; k < r; ++k) {
        const float pk = P[int64_t(k) * m + row];
        float qk[8];
        dev::Vec8<float>::load(Q + int64_t(k) * n + col, qk);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = __fmaf_rn(pk, qk[j], acc[j]);
      }
    }
    const int64_t i = int64_t(row) * n + col;
    float x[8], o[8];
    dev::Vec8<__nv_bfloat16>::load(mef + i, x);
    // the error memory must see the value as the bucket will hold it (rounded to the bucket's type)
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = dev::Vec16<T>::to_float(dev::Vec16<T>::from_float(acc[j]));
    dev::Vec8<T>::store(grad + i, o);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] -= o[j];
    dev::Vec8<__nv_bfloat16>::store(ef + i, x);
  }
}

// ---- cross-rank mean of a (rows x 16) factor + orthonormalisation ----------------------------------------
// One thread-block CLUSTER of kXCtas CTAs per rank; every CTA owns a slice of the rows. local: this
// rank's factor as the GEMM leaves it (rows x 16 fp32, row-major, columns >= r ignored). Everything after
// that is COLUMN-major (element (row, c) at [c * rows + row]) so that every pass is a coalesced stream:
// mean_out (16 x rows fp32): the averaged factor, orthonormalised in place when orth_mean != 0;
// t_out (16 x rows bf16): the orthonormalised averaged factor (rows r..15 zero): the B operand of the
// next GEMM.
// Orthonormalisation is Gram-Schmidt through the Gram matrix (Q = W R^-1 with R^T R = W^T W, the
// Cholesky factor), applied twice ("CholeskyQR2"): each round is one pass that accumulates the r x r Gram
// matrix, a cluster-wide sum over distributed shared memory in a fixed order (every CTA gets the same
// bits), a factorisation done redundantly by one warp of every CTA, and one pass that applies R^-1. A column
// whose pivot vanishes (rank-deficient factor) becomes zero, as a column of norm 0 stays in classical
// Gram-Schmidt. The second round removes the orthogonality loss of the first.
//
// Bound by latency: the factor is a few hundred rows of r values per CTA, which stay in shared memory from the mean to the
// results (a factor too tall for that is worked on in memory, SMEM = false), so that between the flags and the results there are
// two cluster barriers and two factorisations per launch and no trip to L2. Measured on B200, rank 4, 2048 rows: 23.5 -> 9.9 us;
// rank 8 (four factors of 512 to 4608 rows at once): 72 -> 18 us each. Before, every pass went through memory, and one thread
// factorised with its matrices in local memory.
// A rank on its own reads the factor where the GEMM left it. The GEMM then needs no counters, no second look at its tiles and no flag (11 -> 5.5 us), and
// with every kernel of the chain set up while the one before it ends, the four matrices of a ResNet-50 bucket (2.4 to 1.0 M elements, rank 4) take 48 us and not 67.
// With several ranks (one rank of two, four, eight timed, the others' words there already; the same bucket): 92, 102, 124 us with a kernel behind the other and
// the mean taken a column at a time; 84, 97, 122 so (rank 8: 110, 120, 149 -> 94, 107, 138).
constexpr int kXCtas = 8;
constexpr int kXThreads = 512;
constexpr int kXWarps = kXThreads / 32;

// Factorises the Gram matrix in `gram` (lower triangle, packed) and leaves R^-1 (upper triangular) in `rinv`. One warp: lane i holds row
// i of the matrix, columns are eliminated one after the other; then lane c solves for column c of the inverse.
template <int RMAX>
__device__ __forceinline__ void factorise(const float* gram, int r, float (*L)[kCols], float (*rinv)[kCols]) {
  const int lane = threadIdx.x & 31;
  const int row = lane < RMAX ? lane : 0;
  float g[RMAX], diag = 0.0f;
#pragma unroll
  for (int j = 0; j < RMAX; ++j) {
    g[j] = j <= row && row < r ? gram[row * (row + 1) / 2 + j] : 0.0f;
    if (j == row) diag = g[j];
  }
  uint32_t dead = 0;
#pragma unroll
  for (int c = 0; c < RMAX; ++c) {
    if (c < r) {
      const float pivot = __shfl_sync(0xffffffffu, g[c], c), d0 = __shfl_sync(0xffffffffu, diag, c);
      const bool gone = !(pivot > 1e-20f) || !(pivot > 1e-7f * d0);  // pivot vanished: dependent (or zero) column
      const float root = gone ? 1.0f : sqrtf(pivot);
      if (gone) dead |= 1u << c;
      const float l = row == c ? root : gone || row < c ? 0.0f : g[c] / root;
      g[c] = l;
#pragma unroll
      for (int j = c + 1; j < RMAX; ++j) {
        const float lj = __shfl_sync(0xffffffffu, l, j);
        if (j <= row) g[j] = __fmaf_rn(-l, lj, g[j]);
      }
    }
  }
  if (lane < RMAX) {
#pragma unroll
    for (int j = 0; j < RMAX; ++j) L[lane][j] = j <= lane ? g[j] : 0.0f;
  }
  __syncwarp();
  // X = R^-1 where R = L^T (upper triangular): X[j][c] for j <= c; a dead column is zero, and nothing depends on a dead row
  if (lane < RMAX) {
    const int c = lane;
    float x[RMAX];
#pragma unroll
    for (int j = RMAX - 1; j >= 0; --j) {
      float v = 0.0f;
      if (c < r && j <= c && !((dead >> c) & 1u) && !((dead >> j) & 1u)) {
        if (j == c) {
          v = 1.0f / L[c][c];
        } else {
          float sum = 0.0f;
#pragma unroll
          for (int k = RMAX - 1; k > j; --k)
            if (k <= c) sum = __fmaf_rn(L[k][j], x[k], sum);  // R[j][k] = L[k][j]
          v = -sum / L[j][j];
        }
      }
      x[j] = v;
      rinv[j][c] = v;
    }
  }
}

// RMAX: compile-time bound on the rank (4, 8 or 16). SMEM: this CTA's rows fit into shared memory. ALONE: nobody to exchange with, the
// factor is read where the GEMM left it, four columns at a time.
template <int RMAX, bool SMEM, bool ALONE>
__global__ void __launch_bounds__(kXThreads) psgd_exchange_kernel(const __grid_constant__ NangilaPsgdExchangeParams p) {
  constexpr int kAcc = RMAX * (RMAX + 1) / 2;
  cg::cluster_group cluster = cg::this_cluster();
  const int g = int(cluster.block_rank());
  const int vr = blockIdx.x / kXCtas;
  const int me = p.rank0 + vr;
  const int W = p.world, rows = p.rows, r = p.rank;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t slot_bytes = (uint64_t(rows) * r * 4 + 255) & ~uint64_t(255);
  follow();
  const uint32_t epoch = p.epoch_dev != nullptr ? *p.epoch_dev : p.epoch;
  const uint64_t base = p.recv_off + uint64_t(epoch & 1u) * W * slot_bytes;  // two slot sets, by launch parity
  uint32_t* status = p.status[vr];
  const float* local = p.local[vr];
  float* mean = p.mean_out[vr];
  __nv_bfloat16* t_out = static_cast<__nv_bfloat16*>(p.t_out[vr]);
  // this CTA's rows
  const int per = (rows + kXCtas - 1) / kXCtas;
  const int r0 = min(rows, g * per), r1 = min(rows, r0 + per), mine = r1 - r0;
  extern __shared__ float s_rows[];         // [r][per]: the factor's rows, column-major
  __shared__ float s_warp[kXWarps][kAcc];   // per-warp partial sums (summed in warp order: no float atomics)
  __shared__ float s_part[2][kAcc];         // this CTA's partial Gram matrix (lower triangle, packed), one per round
  __shared__ float s_gram[kAcc];            // cluster-wide sum
  __shared__ float s_l[kCols][kCols], s_rinv[kCols][kCols];  // the factor, R^-1 (upper triangular)
  __shared__ int s_ok;

  // 1. store my rows of my factor (r columns, column-major) into every rank's slot [me] (unless the GEMM's
  //    epilogue has done that already)
  if (!ALONE && p.pushed == 0) {
    for (int d = 0; d < W; ++d) {
      float* dst = reinterpret_cast<float*>(p.region[(me + d) % W] + base + uint64_t(me) * slot_bytes);
      for (int c = 0; c < r; ++c)
        for (int i = r0 + tid; i < r1; i += kXThreads) dst[int64_t(c) * rows + i] = local[int64_t(i) * kCols + c];
    }
    __threadfence_system();
    cluster.sync();
    if (g == 0 && tid < W) {
      __threadfence_system();
      st_release_sys(reinterpret_cast<uint32_t*>(p.region[tid] + p.flag_off) + me, epoch);
    }
  }
  // 2. wait for every rank's factor (every CTA polls for itself; on failure all of them still take part in
  //    the cluster barriers below, doing no work)
  if (tid == 0) s_ok = 1;
  __syncthreads();
  if (!ALONE && tid < W) {
    if (!wait_flag(reinterpret_cast<const uint32_t*>(p.region[me] + p.flag_off) + tid, epoch, p.timeout_ns, status,
                   kTimeoutPhase2, uint32_t(me), uint32_t(tid), 8u, 0u))
      s_ok = 0;
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  if (p.orth_mean != 0) may_follow();  // a GEMM of a few CTAs comes next; the reconstruction after the other exchange would fill the device
  // 3. mean in rank order (identical on every rank); columns >= r are zero
  float* work = SMEM ? s_rows : (p.orth_mean ? mean : p.scratch[vr]) + r0;
  const int pitch = SMEM ? per : rows;  // element (row r0 + i, c) at work[c * pitch + i]
  if (ok) {
    const float inv_w = 1.0f / float(W);
    if constexpr (ALONE) {
      for (int i = tid; i < mine; i += kXThreads) {
        const float4* row = reinterpret_cast<const float4*>(local + int64_t(r0 + i) * kCols);
#pragma unroll
        for (int c4 = 0; c4 < RMAX; c4 += 4) {
          if (c4 < r) {
            const float4 q = __ldcg(row + c4 / 4);
            const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (c4 + k < r) {
                if (!p.orth_mean) mean[int64_t(c4 + k) * rows + r0 + i] = v[k];
                work[int64_t(c4 + k) * pitch + i] = v[k];
              }
            }
          }
        }
      }
    } else {
      // (all columns' loads of a few ranks on their way together)
      const float* slots = reinterpret_cast<const float*>(p.region[me] + base) + r0;
      const int64_t slot = int64_t(slot_bytes / 4);
      for (int i = tid; i < mine; i += kXThreads) {
        float acc[RMAX];
#pragma unroll
        for (int c = 0; c < RMAX; ++c) acc[c] = 0.0f;
#pragma unroll 4
        for (int src = 0; src < W; ++src)
#pragma unroll
          for (int c = 0; c < RMAX; ++c)
            if (c < r) acc[c] += slots[src * slot + int64_t(c) * rows + i];
#pragma unroll
        for (int c = 0; c < RMAX; ++c) {
          if (c < r) {
            if (!p.orth_mean) mean[int64_t(c) * rows + r0 + i] = acc[c] * inv_w;
            work[int64_t(c) * pitch + i] = acc[c] * inv_w;
          }
        }
      }
    }
    for (int c = r; c < kCols; ++c)
      for (int i = r0 + tid; i < r1; i += kXThreads) {
        mean[int64_t(c) * rows + i] = 0.0f;
        t_out[int64_t(c) * rows + i] = __float2bfloat16_rn(0.0f);
      }
  }
  // 4. two rounds of Cholesky-QR on `work`
  for (int round = 0; round < 2; ++round) {
    if constexpr (RMAX <= 8) {
      // every thread works on whole rows of its own: all pair products of a row come from registers
      float acc[kAcc];
#pragma unroll
      for (int q = 0; q < kAcc; ++q) acc[q] = 0.0f;
      if (ok) {
        for (int i = tid; i < mine; i += kXThreads) {
          float w[RMAX];
#pragma unroll
          for (int c = 0; c < RMAX; ++c) w[c] = c < r ? work[int64_t(c) * pitch + i] : 0.0f;
          int q = 0;
#pragma unroll
          for (int c = 0; c < RMAX; ++c)
#pragma unroll
            for (int j = 0; j <= c; ++j, ++q) acc[q] = __fmaf_rn(w[c], w[j], acc[q]);
        }
      }
      warp_sums(acc, [&](int q, float v) { s_warp[warp][q] = v; });
    } else {
      // 136 sums are too many for a thread's registers: a warp's lanes share them out, and each lane walks the warp's rows
      __syncthreads();  // rows of other threads: the pass before this one has written them
      for (int q = lane; q < kAcc; q += 32) {
        int c = 0;
        while ((c + 1) * (c + 2) / 2 <= q) ++c;
        const int j = q - c * (c + 1) / 2;
        float v = 0.0f;
        if (ok && c < r)
          for (int i = warp; i < mine; i += kXWarps) v = __fmaf_rn(work[int64_t(c) * pitch + i], work[int64_t(j) * pitch + i], v);
        s_warp[warp][q] = v;
      }
    }
    __syncthreads();
    for (int q = tid; q < kAcc; q += kXThreads) {
      float v = 0.0f;
#pragma unroll
      for (int w = 0; w < kXWarps; ++w) v += s_warp[w][q];  // fixed order: the same bits on every rank
      s_part[round][q] = v;
    }
    cluster.sync();  // every CTA's partial matrix is complete
    for (int q = tid; q < kAcc; q += kXThreads) {
      float part[kXCtas], v = 0.0f;
#pragma unroll
      for (int b = 0; b < kXCtas; ++b) part[b] = *cluster.map_shared_rank(&s_part[round][q], b);
#pragma unroll
      for (int b = 0; b < kXCtas; ++b) v += part[b];  // fixed order
      s_gram[q] = v;
    }
    __syncthreads();
    if (warp == 0) factorise<RMAX>(s_gram, r, s_l, s_rinv);
    __syncthreads();
    if (ok) {
      for (int i = tid; i < mine; i += kXThreads) {
        float w[RMAX];
#pragma unroll
        for (int c = 0; c < RMAX; ++c) w[c] = c < r ? work[int64_t(c) * pitch + i] : 0.0f;
#pragma unroll
        for (int c = 0; c < RMAX; ++c) {
          if (c < r) {
            float o = 0.0f;
#pragma unroll
            for (int j = 0; j <= c; ++j) o = __fmaf_rn(w[j], s_rinv[j][c], o);
            if (round == 0) {
              work[int64_t(c) * pitch + i] = o;
            } else {
              // 5. the results: the orthonormal factor where it is the mean's, and its bf16 copy for the next GEMM's B operand
              const int64_t at = int64_t(c) * rows + r0 + i;
              if (p.orth_mean) mean[at] = o;
              t_out[at] = __float2bfloat16_rn(o);
            }
          }
        }
      }
    }
  }
  cluster.sync();  // a neighbour may still be reading this CTA's part of the last sum
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess) f = nullptr;
    return reinterpret_cast<EncodeFn>(f);
  }();
  return fn;
}
// bf16 matrix with `inner` contiguous elements per row, `outer` rows, row pitch in elements.
bool make_map(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t pitch_elems, uint32_t box_inner,
              uint32_t box_outer) {
  EncodeFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {pitch_elems * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int pick_splits(int tiles, int k_total) {
  int want = 148 / (tiles > 0 ? tiles : 1);
  int max_splits = (k_total + 4 * kSlabK - 1) / (4 * kSlabK);  // at least four slabs per split
  int s = want < 1 ? 1 : (want > max_splits ? max_splits : want);
  return s < 1 ? 1 : s;
}

}  // namespace
}  // namespace nangila

// out (rows x 16 fp32) = M * Bt^T  (transposed = 0: M is m x n, rows = m, contraction over n;
// transposed = 1: out = M^T * Bt^T, rows = n, contraction over m). Bt is 16 x K bf16, K contiguous.
// `out` must be zero-filled when the launch splits K (it always may: zero it).
extern "C" int nangila_psgd_gemm(const void* M, int32_t m, int32_t n, const void* Bt, int32_t transposed, float* out,
                                 uint32_t* status, uint64_t timeout_ns, cudaStream_t stream) {
  return nangila_psgd_gemm_push(M, m, n, Bt, transposed, out, nullptr, status, timeout_ns, stream);
}

static int launch_gemm(const void* M, int32_t m, int32_t n, const void* Bt, int32_t transposed, float* out, int32_t columns,
                       const NangilaPsgdPush* push_in, uint32_t* status, uint64_t timeout_ns, cudaStream_t stream);

extern "C" int nangila_psgd_gemm_columns(const void* M, int32_t m, int32_t n, const void* Bt, int32_t transposed, float* out, int32_t columns,
                                         uint32_t* status, uint64_t timeout_ns, cudaStream_t stream) {
  if (columns < 1 || columns > 16) return int(cudaErrorInvalidValue);
  return launch_gemm(M, m, n, Bt, transposed, out, columns, nullptr, status, timeout_ns, stream);
}

extern "C" int nangila_psgd_gemm_push(const void* M, int32_t m, int32_t n, const void* Bt, int32_t transposed, float* out,
                                      const NangilaPsgdPush* push_in, uint32_t* status, uint64_t timeout_ns,
                                      cudaStream_t stream) {
  return launch_gemm(M, m, n, Bt, transposed, out, push_in != nullptr ? push_in->rank : 16, push_in, status, timeout_ns, stream);
}

static int launch_gemm(const void* M, int32_t m, int32_t n, const void* Bt, int32_t transposed, float* out, int32_t columns,
                       const NangilaPsgdPush* push_in, uint32_t* status, uint64_t timeout_ns, cudaStream_t stream) {
  using namespace nangila;
  NangilaPsgdPush push;
  std::memset(&push, 0, sizeof push);
  if (push_in != nullptr) {
    push = *push_in;
    if (push.counters == nullptr || push.world < 1 || push.world > NANGILA_MAX_RANKS || push.me < 0 || push.me >= push.world ||
        push.rank < 1 || push.rank > 16 || (push.epoch == 0 && push.epoch_dev == nullptr))
      return int(cudaErrorInvalidValue);
    for (int r = 0; r < push.world; ++r)
      if (push.region[r] == nullptr) return int(cudaErrorInvalidValue);
  }
  if (!M || !Bt || !out || !status || m <= 0 || n <= 0 || (n % 8) != 0 || (m % 8) != 0 ||
      (reinterpret_cast<uintptr_t>(M) & 15u) || (reinterpret_cast<uintptr_t>(Bt) & 15u) ||
      (reinterpret_cast<uintptr_t>(out) & 15u))
    return int(cudaErrorInvalidValue);
  CUtensorMap tmA, tmB;
  const int rows = transposed ? n : m;
  const int k_total = transposed ? m : n;
  bool ok;
  if (transposed) ok = make_map(&tmA, M, uint64_t(n), uint64_t(m), uint64_t(n), 64, 64);   // inner = output rows
  else ok = make_map(&tmA, M, uint64_t(n), uint64_t(m), uint64_t(n), 64, 128);             // inner = K
  ok = ok && make_map(&tmB, Bt, uint64_t(k_total), 16, uint64_t(k_total), 64, 16);
  if (!ok) return int(cudaErrorNotSupported);
  const int tiles = (rows + kTileRows - 1) / kTileRows;
  const int splits = pick_splits(tiles, k_total);
  int k_per_split = (k_total + splits - 1) / splits;
  k_per_split = (k_per_split + kSlabK - 1) / kSlabK * kSlabK;
  const int nsplit = (k_total + k_per_split - 1) / k_per_split;
  const dim3 grid{unsigned(tiles), unsigned(nsplit), 1u};
  auto* kernel = transposed ? psgd_gemm_kernel<true> : psgd_gemm_kernel<false>;
  static bool opted_in[2] = {false, false};  // shared memory above the default limit
  if (!opted_in[transposed ? 1 : 0]) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
    opted_in[transposed ? 1 : 0] = true;
  }
  return int(launch_following(kernel, grid, kGemmThreads, kGemmSmem, stream, tmA, tmB, out, rows, k_total, k_per_split, int(nsplit > 1),
                              int(columns), status, timeout_ns, push));
}

extern "C" int nangila_psgd_prep(const void* grad, int32_t dtype, const void* ef, void* mef, int64_t numel, float* z0,
                                 int64_t n0, float* z1, int64_t n1,
                                 cudaStream_t stream) {
  using namespace nangila;
  if (!grad || !ef || !mef || numel <= 0) return int(cudaErrorInvalidValue);
  const int blocks = int(std::min<int64_t>((numel + 2047) / 2048, 148 * 32));
  auto* e = static_cast<const __nv_bfloat16*>(ef);
  auto* o = static_cast<__nv_bfloat16*>(mef);
  switch (dtype) {
    case NANGILA_F32: psgd_prep_kernel<float><<<blocks, 256, 0, stream>>>(static_cast<const float*>(grad), e, o, numel, z0, n0, z1, n1); break;
    case NANGILA_BF16: psgd_prep_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(grad), e, o, numel, z0, n0, z1, n1); break;
    case NANGILA_F16: psgd_prep_kernel<__half><<<blocks, 256, 0, stream>>>(static_cast<const __half*>(grad), e, o, numel, z0, n0, z1, n1); break;
    default: return int(cudaErrorInvalidValue);
  }
  return int(cudaGetLastError());
}

extern "C" int nangila_psgd_reconstruct(void* grad, int32_t dtype, void* ef, const void* mef, const float* P,
                                        const float* Q, int32_t m, int32_t n, int32_t r, cudaStream_t stream) {
  using namespace nangila;
  if (!grad || !ef || !mef || !P || !Q || m <= 0 || n <= 0 || r <= 0 || r > 16) return int(cudaErrorInvalidValue);
  if (n % 8 != 0) return int(cudaErrorInvalidValue);
  const unsigned gx = unsigned((n / 8 + 255) / 256);
  const unsigned gy = unsigned(std::max<int64_t>(1, std::min<int64_t>(m, (148 * 8 + gx - 1) / gx)));
  const dim3 grid{gx, gy};
  auto* e = static_cast<__nv_bfloat16*>(ef);
  cudaError_t err = cudaSuccess;
  auto* f = static_cast<const __nv_bfloat16*>(mef);
#define NANGILA_RECON(T, RQ) err = launch_following(psgd_reconstruct_kernel<T, RQ>, grid, 256, 0, stream, static_cast<T*>(grad), e, f, P, Q, int(m), int(n), int(r))
  switch (dtype) {
    case NANGILA_F32: if (r <= 4) NANGILA_RECON(float, 4); else NANGILA_RECON(float, 0); break;
    case NANGILA_BF16: if (r <= 4) NANGILA_RECON(__nv_bfloat16, 4); else NANGILA_RECON(__nv_bfloat16, 0); break;
    case NANGILA_F16: if (r <= 4) NANGILA_RECON(__half, 4); else NANGILA_RECON(__half, 0); break;
    default: return int(cudaErrorInvalidValue);
  }
#undef NANGILA_RECON
  return int(err);
}

extern "C" uint64_t nangila_psgd_exchange_region_bytes(int32_t rows, int32_t rank, int32_t world, uint64_t* recv_off,
                                                       uint64_t* flag_off) {
  auto align = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
  const uint64_t slot = align(uint64_t(rows) * rank * 4);
  uint64_t off = 0;
  if (recv_off) *recv_off = off;
  off = align(off + 2 * uint64_t(world) * slot);
  if (flag_off) *flag_off = off;
  off = align(off + uint64_t(world) * 4);
  return off;
}

extern "C" int nangila_psgd_exchange(const NangilaPsgdExchangeParams* p, cudaStream_t stream) {
  using namespace nangila;
  if (!p || p->rows <= 0 || p->rank <= 0 || p->rank > 16 || p->world < 1 || p->world > NANGILA_MAX_RANKS || p->nvr < 1 ||
      p->nvr > NANGILA_MAX_VRANKS || (p->nvr > 1 && p->nvr != p->world) || (p->epoch == 0 && p->epoch_dev == nullptr))
    return int(cudaErrorInvalidValue);
  // the CTA's rows stay in shared memory up to this much: with the static part below the default limit of 48 KB
  const size_t rows_bytes = size_t((p->rows + kXCtas - 1) / kXCtas) * size_t(p->rank) * sizeof(float);
  const bool smem = rows_bytes <= 32768;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3{unsigned(p->nvr * kXCtas), 1u, 1u};
  cfg.blockDim = dim3{unsigned(kXThreads), 1u, 1u};
  cfg.dynamicSmemBytes = smem ? rows_bytes : 0;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = kXCtas;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  // several emulated ranks in one launch wait for one another: ask for a cooperative launch so that
  // all their clusters are resident together
  if (p->nvr > 1) {
    attrs[1].id = cudaLaunchAttributeCooperative;
    attrs[1].val.cooperative = 1;
  } else {
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  const NangilaPsgdExchangeParams params = *p;
  // (one rank in the launch: `local` of the group's only rank)
  const bool alone = p->world == 1 && p->pushed == 0 && (reinterpret_cast<uintptr_t>(p->local[0]) & 15u) == 0;
  auto launch = [&](auto rmax) {
    constexpr int R = decltype(rmax)::value;
    auto* kernel = smem ? (alone ? psgd_exchange_kernel<R, true, true> : psgd_exchange_kernel<R, true, false>)
                        : (alone ? psgd_exchange_kernel<R, false, true> : psgd_exchange_kernel<R, false, false>);
    return cudaLaunchKernelEx(&cfg, kernel, params);
  };
  using std::integral_constant;
  const cudaError_t e = p->rank <= 4 ? launch(integral_constant<int, 4>{}) : p->rank <= 8 ? launch(integral_constant<int, 8>{}) : launch(integral_constant<int, kCols>{});
  return int(e);
}
