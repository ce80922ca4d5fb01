// Waits with a limit, for kernels whose warps hand work to one another through mbarriers.  A role whose wait runs out says so in a word that the host can read
// (evo_lost_waits) and ends; the CTA ends once its own copies and products are through, and writes no state.
#pragma once
#include "common.cuh"

namespace evo {

struct WaitLimit { int polls; unsigned int* lost; };      // tries of a wait; the word
int wait_limit(WaitLimit* out);                           // of the calling thread's launches (api.cu)

constexpr int WAIT_POLLS = 1 << 22;

__device__ __forceinline__ bool wait_polls(uint64_t* bar, uint32_t parity, int polls, unsigned int* lost) {
  for (int i = 0; i < polls; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  *(volatile unsigned int*)lost = 1u;
  __threadfence_system();
  return false;
}
__device__ __forceinline__ bool wait_or_give_up(uint64_t* bar, uint32_t parity, const WaitLimit& w) { return wait_polls(bar, parity, w.polls, w.lost); }
// of a whole warp, which stays together: what one lane has lost all have
__device__ __forceinline__ bool warp_wait_or_give_up(uint64_t* bar, uint32_t parity, const WaitLimit& w) {
  for (int i = 0; i < w.polls; ++i)
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  *(volatile unsigned int*)w.lost = 1u;
  __threadfence_system();
  return false;
}
// for what the CTA itself has under way (copies into its shared memory, products): the full limit, whatever the caller's
__device__ __forceinline__ void wait_to_end(uint64_t* bar, uint32_t parity, const WaitLimit& w) { wait_polls(bar, parity, WAIT_POLLS, w.lost); }

}  // namespace evo
