// The meeting of the ranks between two kernels of a collective: what the kernel before it in the stream has stored into peers' memory
// is complete (that kernel has ended), so one word per rank says so, and when every rank's word has arrived the kernel after it
// may read. A launch of one CTA: while it waits for a peer the rest of the GPU belongs to whatever else is queued, the kernels
// around it need no flags, no fences and no residency, and the wait is paid once and not by each of their CTAs (1536 CTAs that each
// looked at four words themselves added 7 us to the reduce-scatter's sum; all of them releasing the words as well, 45 us). All words of the launch's ranks are released before any wait
// begins, so ranks that are emulated in one launch do not depend on one another's progress. A wait that runs out is recorded in the
// rank's status block, which the kernel after it reads first.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "follow.cuh"
#include "nangila_kernels.h"
#include "signal.cuh"

namespace nangila {
namespace comm {

// A launch that holds all ranks of its group (a group of one, ranks emulated on one device) needs no meeting: the end of the kernel before is
// one. What is left of it is a look at the ranks' status blocks by the kernel that reads their data. `status_seen` starts it, a word of one rank
// to a lane; `all_came`, when the data are there (so that it costs no latency), is false on
// all threads of a warp if rank `vr` has failed or another one has, which has then stored nothing (and is reported as one that did not come).
template <typename P>
__device__ __forceinline__ uint32_t status_seen(const P& p) {
  const int lane = int(threadIdx.x) & 31;
  return lane < p.nvr ? *reinterpret_cast<volatile uint32_t*>(&p.status[lane][kStatusCode]) : 0u;
}
template <typename P>
__device__ __forceinline__ bool all_came(const P& p, int vr, uint32_t seen, uint32_t code, uint32_t phase) {
  const uint32_t failed = __ballot_sync(0xffffffffu, seen != 0u);
  if (((failed >> vr) & 1u) != 0u) return false;
  if (failed == 0u || p.nvr != p.world) return true;
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

// P: a parameter block with the members that all exchange kernels share. `ctas`: of the kernel that follows. Where all ranks are in the launch and
// that kernel fits onto the device at once, three launches are what the call costs (reduce-scatter of 16 K to 260 K elements on two to eight ranks: 10 us and
// more, 8 to 9 without the meeting). Larger ones keep it, and so does the all-gather, whose second kernel lost more by the look at all ranks' words (43 -> 50 us).
constexpr int64_t kMeetlessCtas = 8 * 148;
template <typename P>
cudaError_t launch_meet(const P& p, uint64_t flag_off, uint32_t code, uint32_t phase, int64_t ctas, cudaStream_t stream) {
  if (p.nvr == p.world && ctas <= kMeetlessCtas) return cudaSuccess;  // see all_came()
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
