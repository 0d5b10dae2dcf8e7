// Fused Deep-Gradient-Compression exchange for sm_100a: momentum correction, exact top-k threshold
// by radix select, compaction of (index, value) pairs with momentum-factor masking, the sparse
// all-gather over NVLink peer memory and the scatter-accumulate into the dense bucket — one
// cooperative launch per bucket, no NCCL collective.
//
// What it replaces in the reference: DGCCompressor::compress (nangila-core/src/dgc.rs:104-149:
// residual accumulation, top-k by a full sort of |v|, zeroing of the sent entries), decompress
// (:151-174: scatter into zeros) and the all-gather + mean the DDP hook would put around them
// (python/nangila/ddp.py:299-339). Momentum correction and momentum-factor masking are the parts of
// the DGC paper the reference leaves out (dgc.rs:36-38); `momentum = 0` gives the reference's plain
// accumulation.
//
// Phases (grid-wide barriers between them: hardware barriers of a cooperative launch in the single-GPU
// loopback world, counter barriers with a time limit otherwise, see comm/signal.cuh; the launcher clears the scratch words):
//   1  u = m u + g ; v = v + u ; the dense bucket is zeroed. Entries a little below the previous threshold and up, the candidates, are
//      listed, with a histogram of their distance from that bound in steps of 4096 units in the last place
//   2  histogram of the last 12 bits among the candidates of the selected step                   -> threshold bit pattern tau
//   3  compaction: every candidate with |v| >= tau is appended to the send list (bounded by the list capacity), u and v are
//      zeroed there. A group of one rank writes the bucket here and is done
//   4  the list is copied into every rank's receive slot for this rank, then a flag is released
//   5  wait (bounded) for every rank's list, add value / W into the bucket, list by list in rank order
// Without a previous threshold, or if the list does not hold the k largest for sure (fewer than k candidates,
// no room for all of them, a threshold above twice the bound), the threshold comes from a three-pass radix select over
// the dense state (bits [30:20], [19:9], [8:0]; the first histogram is built in phase 1 if there is no previous threshold or it came
// from the dense state itself, and by a CTA whose list is full from there on).
// The selection is exact either way: tau is the k-th largest |v|. Elements equal to tau are all selected, so
// with ties the list can be longer than k (it is cut at the capacity; what is cut stays in v).
//
// What bounds it: phase 1 is HBM (20 bytes an element with a bf16 bucket); what follows is latency, about 2.5 us a barrier and 1.5 to 2
// a selection. Measured on B200, one rank, bf16, copy of the gradient into the bucket included: 13.1 M elements, settled, 73 us (87 with selections that read
// the histograms a word at a time, 195 with phase 1 voting every element and eight barriers). Without that copy, before the selections were
// mended: first step 160 us, the next five, which have no room on the list, 170 to 183; 1.05 M: 52, 57, settled 48.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "launch_util.cuh"
#include "nangila_kernels.h"
#include "quant.cuh"
#include "radix_select.cuh"
#include "signal.cuh"

namespace cg = cooperative_groups;

namespace nangila {
namespace {

using namespace comm;
using namespace rsel;

constexpr int kThreads = 256;

// scratch layout (uint32 words), the first kClearWords cleared before the launch; the candidate list (index, bits pairs) follows
constexpr int kHist0 = 0, kHist1 = kHist0 + kBins0, kHist2 = kHist1 + kBins1;
constexpr int kCursor = kHist2 + kBins2;  // number of selected entries
constexpr int kCandCount = kCursor + 1;   // candidates collected in phase 1, summed over the CTAs
constexpr int kPath = kCursor + 2;        // telemetry: 1 if the selection ran on the list, then the candidates seen
constexpr int kBarrierWord = kCursor + 5;   // counter of the grid barriers of a plain launch
constexpr int kDone = kCursor + 6;          // CTAs that are through (a group of one rank)
constexpr int kSpill = kCursor + 7;         // candidates that found their CTA's segment full
constexpr int kCoarse = kCursor + 8;        // candidates by distance from the bound, kStep apart
constexpr int kStepBits = 12, kCoarseBins = 2048, kFineBins = 1 << kStepBits;
constexpr int kFine = kCoarse + kCoarseBins;  // the selected step's candidates by distance
constexpr int kClearWords = kFine + kFineBins;
// kept from launch to launch (whatever is there at first does no harm): a threshold, the bound for the launch after it, and the threshold
// if it came from the dense state
constexpr int kKept = kClearWords;
constexpr int kScratchWords = kClearWords + 8;
constexpr uint32_t kBand = 4;  // candidates wanted, in multiples of k

template <typename T>
__device__ __forceinline__ float ldf(const T* p, int64_t i) { return dev::Vec16<T>::to_float(p[i]); }

// Four consecutive elements (the bucket and the fp32 state are at least 16-byte aligned and the
// vector index is a multiple of 4, so 8- and 16-byte accesses are aligned).
template <typename T>
__device__ __forceinline__ void ld4(const T* p, int64_t i, float (&x)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = *reinterpret_cast<const float4*>(p + i);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  } else {
    const uint2 a = *reinterpret_cast<const uint2*>(p + i);
    const T* h = reinterpret_cast<const T*>(&a);
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = dev::Vec16<T>::to_float(h[k]);
  }
}
template <typename T>
__device__ __forceinline__ void st4_zero(T* p, int64_t i) {
  if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(p + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  else *reinterpret_cast<uint2*>(p + i) = make_uint2(0u, 0u);
}

// One vote per distinct bin of the warp: gradients cluster in a handful of exponent bins, and 32 lanes
// adding to the same shared-memory word would be serialised. `active` lanes hold a valid `bin`.
__device__ __forceinline__ void hist_add(uint32_t* hist, uint32_t bin, bool active) {
  const uint32_t live = __ballot_sync(0xffffffffu, active);
  if (!active) return;
  const uint32_t peers = __match_any_sync(live, bin);
  if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[bin], uint32_t(__popc(peers)));
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 3) dgc_fused_kernel(const __grid_constant__ NangilaDgcParams p) {
  cg::grid_group grid = cg::this_grid();
  const int vr = blockIdx.y;
  // Grid-wide barriers: the hardware one when several ranks are emulated in one (cooperative) launch; with a
  // real process group a counter barrier over the CTAs of this launch, so the kernel needs no cooperative
  // launch, can start while backward still holds part of the GPU, and runs with a capped number of CTAs.
  const bool coop = p.nvr > 1;
  GridBarrier soft(p.scratch[vr] + kBarrierWord, gridDim.x);
  auto gsync = [&]() -> bool {
    if (coop) {
      grid.sync();
      return true;
    }
    return soft.sync(p.timeout_ns, p.status[vr], uint32_t(p.rank0 + vr), p.epoch);
  };
  const int me = p.rank0 + vr;
  const int W = p.world;
  const int64_t n = p.n;
  T* __restrict__ grad = static_cast<T*>(p.grad[vr]);
  float* __restrict__ u = p.u[vr];
  float* __restrict__ v = p.v[vr];
  uint32_t* scratch = p.scratch[vr];
  uint32_t* status = p.status[vr];
  uint8_t* myreg = p.region[me];
  const uint32_t cap = p.capacity;
  const uint64_t slot_bytes = 16 + uint64_t(cap) * 8;
  // Two sets of receive slots, used alternately by epoch parity: a rank that runs one launch ahead
  // writes the other set while a slower peer may still be scattering from this one; it cannot get
  // two launches ahead because its wait in phase 5 needs the peer's flag of the launch in between.
  const uint64_t recv_base = p.recv_off + uint64_t(p.epoch & 1u) * uint64_t(W) * slot_bytes;
  // local send list lives in this rank's own receive slot for itself
  uint8_t* myslot = myreg + recv_base + uint64_t(me) * slot_bytes;
  uint32_t* my_idx = reinterpret_cast<uint32_t*>(myslot + 16);
  float* my_val = reinterpret_cast<float*>(myslot + 16 + uint64_t(cap) * 4);

  __shared__ uint32_t sh_hist[kBins0], sh_top[kBins0];
  __shared__ uint32_t sh_sel[10];
  __shared__ uint32_t sh_cand_cnt;   // candidates this CTA has found
  __shared__ uint32_t sh_list_full;  // not 0: one of them had no room
  const int64_t tid0 = int64_t(blockIdx.x) * kThreads + threadIdx.x;
  const int64_t stride = int64_t(gridDim.x) * kThreads;
  // The dense passes walk the bucket in groups of 4 elements; every warp keeps all 32 lanes in the loop
  // (the loop bound is rounded up per warp) so that the warp-wide votes below are well defined.
  const int64_t n4 = n / 4;                          // whole groups
  const int64_t groups = (n + 3) / 4;                // including the ragged last one
  const int64_t groups_rounded = (groups + 31) / 32 * 32;

  // Candidates. Between two calls on the same bucket the threshold moves little, so the k largest entries are nearly always among
  // those above a bound a little below the previous threshold, a few thousand to look through instead of the dense state. The bound
  // is 0.96 of the threshold, or the value that 4 k entries were above last time if that is higher: unsent entries pile up just
  // below the threshold, and once the threshold has settled 36 k lie within 4 % of it.
  const uint32_t tau_prev = p.out_count[vr][1];
  const uint32_t cand_cap = p.cand_capacity;
  const bool use_list = cand_cap > 0 && tau_prev > 0 && tau_prev < 0x7f800000u;
  uint32_t cand_thr = 0xffffffffu;  // nothing qualifies
  if (use_list) {
    cand_thr = __float_as_uint(__uint_as_float(tau_prev) * 0.96f);
    if (scratch[kKept] == tau_prev && scratch[kKept + 1] <= tau_prev) cand_thr = max(cand_thr, scratch[kKept + 1]);
  }
  // A launch after one that went over the dense state may well have to do so too (the second to seventh step of a large bucket), with a
  // list that fills up only near the end: it counts top bits from the start, while it collects (67 M fp32 elements, sixth step: 1057 -> 811 us).
  const bool doubt = use_list && scratch[kKept + 2] == tau_prev;
  // Half of the list is cut into a segment per CTA, which fills it without asking anybody; the candidates are not spread evenly (layers
  // have gradients of different size), so what finds its segment full goes to the other half, place by place.
  const uint32_t seg_cap = cand_cap / 2 / gridDim.x;
  const uint32_t spill_cap = cand_cap - seg_cap * gridDim.x;
  uint32_t* cand_idx = scratch + kScratchWords + uint64_t(blockIdx.x) * seg_cap;
  uint32_t* cand_bits = cand_idx + cand_cap;
  uint32_t* spill_idx = scratch + kScratchWords + uint64_t(gridDim.x) * seg_cap;
  uint32_t* spill_bits = spill_idx + cand_cap;

  if (threadIdx.x == 0) sh_cand_cnt = sh_list_full = 0u;

  // ---- phase 1: momentum correction, candidates (or the first histogram) ----
  static_assert(kCoarseBins == kBins0, "cleared together");
  for (int i = threadIdx.x; i < kBins0; i += kThreads) sh_hist[i] = sh_top[i] = 0u;
  __syncthreads();
  // The candidates among a lane's eight entries, from `first` on; all lanes of a warp come here. Space is reserved once for the
  // warp's 256 entries. Where far more entries qualify than the list holds (the first steps of a bucket, gradients that have jumped) the
  // selection goes over the dense state whatever is collected, so a CTA that has found the list full stops: without that, 13.1 M entries
  // that all qualify made as many reservations in one word (455 us a step; 170 to 183 this way, 33 M: 1100 to 1200 and 400 to 430). From
  // there on its warps count bits [30:20] instead, as they do without a previous threshold, so that less is left to be read again.
  // Returns false if the entries were not collected because the list is full.
  volatile uint32_t* list_full = &sh_list_full;
  auto collect = [&](int64_t first, const float (&v_new)[8], int valid) -> bool {
    uint32_t mine = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < valid && (__float_as_uint(v_new[k]) & 0x7fffffffu) >= cand_thr) mine |= 1u << k;
    if (!__any_sync(0xffffffffu, mine != 0u)) return true;
    if (__any_sync(0xffffffffu, *list_full != 0u)) return false;
    const int lane = threadIdx.x & 31;
    uint32_t incl = uint32_t(__popc(mine));
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    uint32_t base = 0, spill = 0;  // the warp's entries get base, base + 1, ...; those from seg_cap on go to spill, spill + 1, ...
    if (lane == 31) {
      base = atomicAdd(&sh_cand_cnt, incl);
      const uint32_t over = base + incl > seg_cap ? base + incl - max(base, seg_cap) : 0u;
      if (over > 0u) {
        spill = atomicAdd(&scratch[kSpill], over);
        if (spill + over > spill_cap) *list_full = 1u;
      }
    }
    base = __shfl_sync(0xffffffffu, base, 31);
    spill = __shfl_sync(0xffffffffu, spill, 31);
    uint32_t pos = base + incl - uint32_t(__popc(mine));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (mine & (1u << k)) {
        const uint32_t b = __float_as_uint(v_new[k]) & 0x7fffffffu;
        if (pos < seg_cap) {
          cand_idx[pos] = uint32_t(first + k);
          cand_bits[pos] = b;
        } else {
          const uint32_t at = spill + (pos - max(base, seg_cap));
          if (at < spill_cap) {
            spill_idx[at] = uint32_t(first + k);
            spill_bits[at] = b;
          }
        }
        atomicAdd(&sh_hist[min((b - cand_thr) >> kStepBits, uint32_t(kCoarseBins - 1))], 1u);
        ++pos;
      }
    }
    return true;
  };
  auto vote_top = [&](const float (&x)[8], int valid) {
#pragma unroll
    for (int k = 0; k < 8; ++k) hist_add(sh_top, (__float_as_uint(x[k]) & 0x7fffffffu) >> 20, k < valid);
  };
  const int64_t n8 = n / 8, groups8 = (n + 7) / 8, groups8_rounded = (groups8 + 31) / 32 * 32;
  bool collecting = use_list;
  int64_t vote_from = use_list && !doubt ? groups8_rounded : 0;  // this lane's groups from here on are in the first histogram (the same iteration for a warp)
  for (int64_t q = tid0; q < groups8_rounded; q += stride) {
    float vn[8];
    int valid = 0;
    if (q < n8) {
      float g[8], uu[8];
      ld4<T>(grad, q * 8, reinterpret_cast<float (&)[4]>(g[0]));
      ld4<T>(grad, q * 8 + 4, reinterpret_cast<float (&)[4]>(g[4]));
      dev::Vec8<float>::load(u + q * 8, uu);
      dev::Vec8<float>::load(v + q * 8, vn);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        uu[k] = __fmaf_rn(p.momentum, uu[k], dev::sanitize(g[k]));
        vn[k] += uu[k];
      }
      dev::Vec8<float>::store(u + q * 8, uu);
      dev::Vec8<float>::store(v + q * 8, vn);
      st4_zero<T>(grad, q * 8);  // the dense result starts from zero
      st4_zero<T>(grad, q * 8 + 4);
      valid = 8;
    } else if (q < groups8) {
      for (int k = 0; k < 8; ++k) {
        const int64_t i = q * 8 + k;
        vn[k] = 0.0f;
        if (i < n) {
          const float un = __fmaf_rn(p.momentum, u[i], dev::sanitize(ldf(grad, i)));
          vn[k] = v[i] + un;
          u[i] = un;
          v[i] = vn[k];
          grad[i] = dev::Vec16<T>::from_float(0.0f);
          valid = k + 1;
        }
      }
    }
    if (collecting && !collect(q * 8, vn, valid)) {
      collecting = false;
      vote_from = min(vote_from, q);
    }
    if (!collecting || doubt) vote_top(vn, valid);
  }
  __syncthreads();
  auto add_top = [&] {
    for (int i = threadIdx.x; i < kBins0; i += kThreads)
      if (sh_top[i]) atomicAdd(&scratch[kHist0 + i], sh_top[i]);
  };
  if (use_list) {
    for (int i = threadIdx.x; i < kCoarseBins; i += kThreads)
      if (sh_hist[i]) atomicAdd(&scratch[kCoarse + i], sh_hist[i]);
  }
  if (!use_list || doubt) add_top();
  const uint32_t my_cand = min(sh_cand_cnt, seg_cap);  // entries of this CTA's segment
  if (threadIdx.x == 0) atomicAdd(&scratch[kCandCount], my_cand);
  if (!gsync()) return;
  uint32_t want = p.k, bin0, bin1, bin2;
  const uint32_t nspill = __ldcg(scratch + kSpill), ncand = __ldcg(scratch + kCandCount) + nspill;
  bool from_list = use_list && ncand >= p.k && nspill <= spill_cap;  // same on every CTA
  uint32_t coarse = 0;
  if (from_list) {
    select_bin<kCoarseBins>(scratch + kCoarse, want, coarse, sh_sel);
    from_list = coarse < uint32_t(kCoarseBins - 1);  // the last one holds everything from there on
  }
  // Appends the entries that the lanes of a warp have selected to the send list, and takes them out of the state.
  const float inv_w = 1.0f / float(W);
  auto append = [&](bool sel, int64_t i) {
    const uint32_t mask = __ballot_sync(0xffffffffu, sel);
    if (mask == 0u) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == __ffs(mask) - 1) base = atomicAdd(&scratch[kCursor], uint32_t(__popc(mask)));
    base = __shfl_sync(0xffffffffu, base, __ffs(mask) - 1);
    if (sel) {
      const uint32_t pos = base + uint32_t(__popc(mask & ((1u << lane) - 1u)));
      if (pos < cap) {
        const float x = v[i];
        my_idx[pos] = uint32_t(i);
        my_val[pos] = x;
        v[i] = 0.0f;
        u[i] = 0.0f;
        if (W == 1) grad[i] = dev::Vec16<T>::from_float(__fmaf_rn(x, inv_w, 0.0f));  // nobody else's entries to add
      }
    }
  };
  // The ranks of a cooperative launch share its barriers but not their choice of path: there, every path passes kSelectSyncs.
  constexpr int kSelectSyncs = 3;
  int select_syncs = 0;
  auto ssync = [&]() -> bool {
    ++select_syncs;
    return gsync();
  };
  auto even_out = [&] {
    if (coop)
      for (; select_syncs < kSelectSyncs; ++select_syncs) grid.sync();
  };
  uint32_t tau;
  if (from_list) {
    // ---- phases 2 and 3 over the candidate list: this CTA scans its own segment ----
    auto count_fine = [&](uint32_t bits) {
      const uint32_t d = bits - cand_thr;
      if ((d >> kStepBits) == coarse) atomicAdd(&scratch[kFine + (d & (kFineBins - 1))], 1u);
    };
    for (uint32_t j = threadIdx.x; j < my_cand; j += kThreads) count_fine(cand_bits[j]);
    for (uint32_t j = uint32_t(tid0); j < nspill; j += uint32_t(stride)) count_fine(__ldcg(spill_bits + j));
    // The next launch's bound, by the first CTA: at the end where nobody waits for that one, with peers here, beside the other CTAs' counting (at
    // the end it costs two emulated ranks of 65 536 elements 1 us in 51).
    uint32_t next_bound = 0;
    auto find_next_bound = [&] {
      uint32_t rank = min(kBand * p.k, ncand), bin;
      select_bin<kCoarseBins>(scratch + kCoarse, rank, bin, sh_sel);
      next_bound = cand_thr + (bin << kStepBits);
    };
    if (blockIdx.x == 0 && W > 1) find_next_bound();
    if (!ssync()) return;
    uint32_t fine;
    select_bin<kFineBins>(scratch + kFine, want, fine, sh_sel);
    tau = cand_thr + (coarse << kStepBits) + fine;
    even_out();
    const uint32_t nc_rounded = (my_cand + 31u) / 32u * 32u;
    for (uint32_t j = threadIdx.x; j < nc_rounded; j += kThreads) {
      const bool sel = j < my_cand && cand_bits[j] >= tau && p.k > 0;
      append(sel, sel ? int64_t(cand_idx[j]) : 0);
    }
    const uint32_t ns_rounded = (nspill + 31u) / 32u * 32u;
    for (uint32_t j = uint32_t(tid0); j < ns_rounded; j += uint32_t(stride)) {
      const bool sel = j < nspill && __ldcg(spill_bits + j) >= tau && p.k > 0;
      append(sel, sel ? int64_t(__ldcg(spill_idx + j)) : 0);
    }
    if (blockIdx.x == 0) {  // every CTA has read the old pair before the first barrier
      if (W == 1) find_next_bound();
      if (threadIdx.x == 0) {
        scratch[kKept] = tau;
        scratch[kKept + 1] = next_bound;
      }
    }
  } else {
    // bit patterns of |v| for one group (0 beyond the end: never selected, never counted)
    auto load_bits = [&](int64_t q, uint32_t (&b)[4]) {
      if (q < n4) {
        const uint4 a = *reinterpret_cast<const uint4*>(v + q * 4);
        b[0] = a.x & 0x7fffffffu; b[1] = a.y & 0x7fffffffu; b[2] = a.z & 0x7fffffffu; b[3] = a.w & 0x7fffffffu;
      } else {
  #pragma unroll
        for (int k = 0; k < 4; ++k) b[k] = (q * 4 + k < n) ? (__float_as_uint(v[q * 4 + k]) & 0x7fffffffu) : 0xffffffffu;
      }
    };

    if (use_list && !doubt) {
      // ---- bits [30:20] of what phase 1 went through while it still collected ----
      for (int64_t q = tid0; q < vote_from; q += stride) {
        float x[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        int valid = 0;
        if (q < n8) {
          dev::Vec8<float>::load(v + q * 8, x);
          valid = 8;
        } else if (q < groups8) {
          valid = int(n - q * 8);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < valid) x[k] = v[q * 8 + k];
        }
        vote_top(x, valid);
      }
      __syncthreads();
      add_top();
      if (!ssync()) return;
    }
    want = p.k;
    select_bin<kBins0>(scratch + kHist0, want, bin0, sh_sel);

    // ---- bits [19:9] ----
    for (int i = threadIdx.x; i < kBins1; i += kThreads) sh_hist[i] = 0u;
    __syncthreads();
    for (int64_t q = tid0; q < groups_rounded; q += stride) {
      uint32_t b[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
      if (q < groups) load_bits(q, b);
  #pragma unroll
      for (int k = 0; k < 4; ++k) hist_add(sh_hist, (b[k] >> 9) & 0x7ffu, b[k] != 0xffffffffu && (b[k] >> 20) == bin0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins1; i += kThreads)
      if (sh_hist[i]) atomicAdd(&scratch[kHist1 + i], sh_hist[i]);
    if (!ssync()) return;
    select_bin<kBins1>(scratch + kHist1, want, bin1, sh_sel);

    // ---- bits [8:0] ----
    for (int i = threadIdx.x; i < kBins2; i += kThreads) sh_hist[i] = 0u;
    __syncthreads();
    const uint32_t prefix = (bin0 << 11) | bin1;
    for (int64_t q = tid0; q < groups_rounded; q += stride) {
      uint32_t b[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
      if (q < groups) load_bits(q, b);
  #pragma unroll
      for (int k = 0; k < 4; ++k) hist_add(sh_hist, b[k] & 0x1ffu, b[k] != 0xffffffffu && (b[k] >> 9) == prefix);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins2; i += kThreads)
      if (sh_hist[i]) atomicAdd(&scratch[kHist2 + i], sh_hist[i]);
    if (!ssync()) return;
    select_bin<kBins2>(scratch + kHist2, want, bin2, sh_sel);
    tau = (prefix << 9) | bin2;  // bit pattern of the k-th largest |v|
    if (blockIdx.x == 0 && threadIdx.x == 0) scratch[kKept + 2] = tau;

    even_out();

    // ---- phase 3: compaction ----
    for (int64_t q = tid0; q < groups_rounded; q += stride) {
      uint32_t b[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
      if (q < groups) load_bits(q, b);
#pragma unroll
      for (int k = 0; k < 4; ++k) append(b[k] != 0xffffffffu && b[k] >= tau && (p.k > 0) && b[k] != 0u, q * 4 + k);
    }
  }
  auto publish = [&](uint32_t count) {
    *reinterpret_cast<uint32_t*>(myslot) = count;
    p.out_count[vr][0] = count;
    p.out_count[vr][1] = tau;
    scratch[kPath] = from_list ? 1u : 0u;
    scratch[kPath + 1] = ncand;
  };
  if (W == 1) {
    // the bucket is complete; the CTA that ends last knows how many entries there were
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(&scratch[kDone], 1u) == gridDim.x - 1) {
        __threadfence();
        publish(min(__ldcg(scratch + kCursor), cap));
        st_release_sys(reinterpret_cast<uint32_t*>(myreg + p.flag_off) + me, p.epoch);
      }
    }
    return;
  }
  if (!gsync()) return;
  const uint32_t count = min(scratch[kCursor], cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) publish(count);

  // ---- phase 4: copy the list into every other rank's slot for this rank, release flags ----
  for (int d = 1; d < W; ++d) {
    const int r = (me + d) % W;
    uint8_t* dst = p.region[r] + recv_base + uint64_t(me) * slot_bytes;
    uint32_t* d_idx = reinterpret_cast<uint32_t*>(dst + 16);
    float* d_val = reinterpret_cast<float*>(dst + 16 + uint64_t(cap) * 4);
    for (int64_t j = tid0; j < count; j += stride) {
      d_idx[j] = my_idx[j];
      d_val[j] = my_val[j];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<uint32_t*>(dst) = count;
  }
  __threadfence_system();
  if (!gsync()) return;
  if (blockIdx.x == 0 && threadIdx.x < W) {
    __threadfence_system();
    st_release_sys(reinterpret_cast<uint32_t*>(p.region[threadIdx.x] + p.flag_off) + me, p.epoch);
  }

  // ---- phase 5: wait for every rank's list and accumulate it ----
  // The lists are added in rank order with a grid barrier after each, so every rank performs the same
  // floating-point additions in the same order and all replicas end up with identical bits. Indices
  // inside one list are unique, so no atomics are needed. A CTA whose wait fails keeps taking part in
  // the barriers (skipping the work) so that nobody is left waiting for it.
  bool alive = true;
  for (int r = 0; r < W; ++r) {
    bool ok = true;
    if (alive && threadIdx.x == 0)
      ok = wait_flag(reinterpret_cast<const uint32_t*>(myreg + p.flag_off) + r, p.epoch, p.timeout_ns, status,
                     kTimeoutPhase2, uint32_t(me), uint32_t(r), 6u, 0u);
    alive = __syncthreads_and(ok ? 1 : 0) && alive;
    if (alive) {
      const uint8_t* src = myreg + recv_base + uint64_t(r) * slot_bytes;
      const uint32_t cnt = min(*reinterpret_cast<const uint32_t*>(src), cap);
      const uint32_t* s_idx = reinterpret_cast<const uint32_t*>(src + 16);
      const float* s_val = reinterpret_cast<const float*>(src + 16 + uint64_t(cap) * 4);
      for (int64_t j = tid0; j < cnt; j += stride) {
        const uint32_t idx = s_idx[j];
        if (idx < n) grad[idx] = dev::Vec16<T>::from_float(__fmaf_rn(s_val[j], inv_w, ldf(grad, idx)));
      }
    }
    if (!gsync()) return;
  }
}

}  // namespace
}  // namespace nangila

extern "C" uint64_t nangila_dgc_region_bytes(uint32_t capacity, int32_t world, uint64_t* recv_off, uint64_t* flag_off) {
  auto align = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
  uint64_t off = 0;
  if (recv_off) *recv_off = off;
  off = align(off + 2 * uint64_t(world) * (16 + uint64_t(capacity) * 8));
  if (flag_off) *flag_off = off;
  off = align(off + uint64_t(world) * 4);
  return off;
}

extern "C" uint32_t nangila_dgc_scratch_words(void) { return nangila::kScratchWords; }

extern "C" int nangila_dgc_launch(const NangilaDgcParams* p, cudaStream_t stream) {
  using namespace nangila;
  if (p == nullptr || p->n <= 0 || p->n > 0x7fffffffll || p->world < 1 || p->world > NANGILA_MAX_RANKS ||
      p->nvr < 1 || p->nvr > NANGILA_MAX_VRANKS || p->rank0 < 0 || p->rank0 + p->nvr > p->world ||
      (p->nvr > 1 && p->nvr != p->world) || p->epoch == 0 || p->capacity == 0 ||
      p->capacity % 4 != 0 || p->k > p->capacity || (p->cand_capacity != 0 && p->cand_capacity < p->k) || !(p->momentum >= 0.0f && p->momentum < 1.0f))
    return int(cudaErrorInvalidValue);
  const void* fn;
  switch (p->grad_dtype) {
    case NANGILA_F32: fn = reinterpret_cast<const void*>(&dgc_fused_kernel<float>); break;
    case NANGILA_BF16: fn = reinterpret_cast<const void*>(&dgc_fused_kernel<__nv_bfloat16>); break;
    case NANGILA_F16: fn = reinterpret_cast<const void*>(&dgc_fused_kernel<__half>); break;
    default: return int(cudaErrorInvalidValue);
  }
  int grid_x = 0;
  const cudaError_t ce = clamp_grid(fn, kThreads, 0, p->grid_x, p->nvr, &grid_x);
  if (ce != cudaSuccess) return int(ce);
  dim3 grid(unsigned(grid_x), unsigned(p->nvr)), block(kThreads);
  void* args[] = {const_cast<NangilaDgcParams*>(p)};
  // histograms, cursors and the counter of the in-kernel grid barrier start from zero
  for (int v = 0; v < p->nvr; ++v) {
    const cudaError_t me = cudaMemsetAsync(p->scratch[v], 0, sizeof(uint32_t) * kClearWords, stream);
    if (me != cudaSuccess) return int(me);
  }
  if (p->nvr > 1) return int(cudaLaunchCooperativeKernel(fn, grid, block, args, 0, stream));
  // real process group: plain launch
  return int(cudaLaunchKernel(fn, grid, block, args, 0, stream));
}
