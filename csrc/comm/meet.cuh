// The meeting of the ranks between two kernels of a collective: what the first has stored into peers' memory is complete when that kernel has ended, so one
// word per rank says so, and when every rank's word has arrived the second may read. A wait that runs out is recorded in the rank's status block.
// Where they meet depends on the launch (how_to_meet):
//   a kernel between the two, of one CTA: while it waits for a peer the rest of the GPU belongs to whatever else is queued, and the wait is paid once and
//     not by each CTA of the second kernel (1536 CTAs that each looked at four words themselves added 7 us to the reduce-scatter's sum; all of them
//     releasing the words as well, 45 us).
//   the second kernel itself, where it has few CTAs: a third launch is what a small call costs.
//   nowhere, where all ranks of the group are in the launch (a group of one, ranks emulated on one device): the end of the first kernel is the meeting.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "follow.cuh"
#include "nangila_kernels.h"
#include "signal.cuh"

namespace nangila {
namespace comm {

enum Met { kMetBefore, kMetInLaunch, kMeetHere };  // in a kernel of its own, or there is only one rank; all ranks are in the launch; in the kernel that reads

// In the kernel that reads, when the one before it is complete (and so is what it has stored, at the peers' too): false, on all threads, if
// this rank has failed or a rank does not come. `seen` starts the look at a status block, for all_came().
template <Met MET, typename P>
__device__ __forceinline__ bool arrive(const P& p, int vr, uint64_t flag_off, uint32_t code, uint32_t phase, uint32_t& seen) {
  if constexpr (MET == kMeetHere) {
    const int me = p.rank0, r = int(threadIdx.x);
    const bool peer = r < p.world && r != me;
    const uint32_t* word = reinterpret_cast<const uint32_t*>(p.region[me] + flag_off) + r;
    // (both loads on their way together; most words are there by now)
    const uint32_t failed = *reinterpret_cast<volatile uint32_t*>(&p.status[0][kStatusCode]);
    const bool there = !peer || epoch_reached(ld_acquire_sys(word), p.epoch);
    // a rank that has failed before has stored nothing: its word stays away, and the others' waits for it run out
    if (peer && failed == 0u && blockIdx.x == 0 && blockIdx.y == 0) st_release_sys(reinterpret_cast<uint32_t*>(p.region[r] + flag_off) + me, p.epoch);
    __syncthreads();  // the words are on their way to all ranks before any wait begins
    const bool ok = failed == 0u && (there || wait_flag(word, p.epoch, p.timeout_ns, p.status[0], code, uint32_t(me), uint32_t(r), phase, 0u));
    return __syncthreads_and(ok ? 1 : 0) != 0;
  } else if constexpr (MET == kMetInLaunch) {  // a word of one rank to a lane
    const int lane = int(threadIdx.x) & 31;
    seen = lane < p.nvr ? *reinterpret_cast<volatile uint32_t*>(&p.status[lane][kStatusCode]) : 0u;
    return true;
  } else {
    seen = *reinterpret_cast<volatile uint32_t*>(&p.status[vr][kStatusCode]);
    return true;
  }
}
// When the data are there, so that the look costs no latency: false, on all threads of a warp, if this rank has failed, or another one of the launch
// has, which has then stored nothing (and is reported as one that did not come).
template <Met MET, typename P>
__device__ __forceinline__ bool all_came(const P& p, int vr, uint32_t seen, uint32_t code, uint32_t phase) {
  if constexpr (MET == kMeetHere) return true;
  if constexpr (MET == kMetBefore) return seen == 0u;
  const uint32_t failed = __ballot_sync(0xffffffffu, seen != 0u);
  if (((failed >> vr) & 1u) != 0u) return false;
  if (failed == 0u) return true;
  if (threadIdx.x == 0)
    report_failure(p.status[vr], code, uint32_t(p.rank0 + vr), uint32_t(p.rank0 + __ffs(failed) - 1), p.epoch, 0u, phase, blockIdx.x);
  return false;
}

struct MeetArgs {
  uint8_t* region[NANGILA_MAX_RANKS];
  uint32_t* status[NANGILA_MAX_VRANKS];
  uint64_t flag_off;  // of the words, one per rank, in every region
  uint64_t timeout_ns;
  int32_t world, rank0, nvr;
  uint32_t epoch, code, phase;
};
constexpr int kMeetThreads = NANGILA_MAX_RANKS * NANGILA_MAX_VRANKS;

static __global__ void __launch_bounds__(kMeetThreads) meet_kernel(const __grid_constant__ MeetArgs a) {
  follow();
  const int v = int(threadIdx.x) / a.world, r = int(threadIdx.x) % a.world;
  // a rank that has failed before has stored nothing: its word stays away, and the others' waits for it run out
  const bool sound = v < a.nvr && *reinterpret_cast<volatile uint32_t*>(&a.status[v][kStatusCode]) == 0u;
  if (sound) st_release_sys(reinterpret_cast<uint32_t*>(a.region[r] + a.flag_off) + a.rank0 + v, a.epoch);
  __syncthreads();
  if (sound)
    wait_flag(reinterpret_cast<const uint32_t*>(a.region[a.rank0 + v] + a.flag_off) + r, a.epoch, a.timeout_ns, a.status[v], a.code,
              uint32_t(a.rank0 + v), uint32_t(r), a.phase, 0u);
}

// Where the ranks meet; `ctas`: of the kernel that reads. us a call, 131 072 bf16 elements a rank. One rank of a group of eight, the others' words
// there already: all-gather 10.2 with the kernel in between, 6.9 without (and tiles of one iteration, fsdp_ag_dequant.cu; one kernel with a flag per
// chunk: 9.0), reduce-scatter 10.4 and 8.3 (15.3). Four emulated ranks: 10.3 and 7.2, 10.7 and 8.1.
//   CTAs that wait for a peer keep other kernels off the SMs: two an SM, not more.
//   The look at all ranks' words costs every CTA a read, more where it has little else to do (`most_in_launch`, by the caller's kernel). With the kernel in
//   between / without: all-gather of 4 x 262 144 bf16 elements (384 CTAs) 10.4 / 8.4; INT4, 8 x 131 072 fp32 (896 CTAs) 18.7 / 20.2, 4 x 786 432 bf16 (1152)
//   15.1 / 15.5. Reduce-scatter of 4 x 1.6 M (768) 26.8 / 24.9; the look without need for it, 4 x 3.1 M a rank (1536): 42.9 / 45.4.
constexpr int64_t kMeetHereCtas = 2 * 148;
template <typename P>
Met how_to_meet(const P& p, int64_t ctas, int64_t most_in_launch) {
  if (p.nvr == p.world) return p.world > 1 && ctas <= most_in_launch ? kMetInLaunch : kMetBefore;
  return p.nvr == 1 && ctas <= kMeetHereCtas ? kMeetHere : kMetBefore;
}
// The kernel in between, if there is one. P: a parameter block with the members that all exchange kernels share.
template <typename P>
cudaError_t launch_meet(const P& p, Met met, uint64_t flag_off, uint32_t code, uint32_t phase, cudaStream_t stream) {
  if (met != kMetBefore || p.world == 1) return cudaSuccess;
  MeetArgs a{};
  for (int r = 0; r < p.world; ++r) a.region[r] = p.region[r];
  for (int v = 0; v < p.nvr; ++v) a.status[v] = p.status[v];
  a.flag_off = flag_off;
  a.timeout_ns = p.timeout_ns;
  a.world = p.world;
  a.rank0 = p.rank0;
  a.nvr = p.nvr;
  a.epoch = p.epoch;
  a.code = code;
  a.phase = phase;
  return launch_following(meet_kernel, dim3(1), kMeetThreads, 0, stream, a);
}

}  // namespace comm
}  // namespace nangila
