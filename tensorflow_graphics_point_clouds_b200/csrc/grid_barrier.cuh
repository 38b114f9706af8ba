// Barrier over blocks of a cooperative launch, with a bounded wait.  The bound is on a
// stall: a block with more work than the others says so (progress).
#pragma once

#include "common.cuh"

namespace tfgpc {

constexpr unsigned kGaveUp = 0x80000000u;    // in a barrier's counter

// Called by one lane between pieces of work of well under half a period.
__device__ __forceinline__ void show_progress(unsigned* progress) { atomicAdd(progress, 1u); }

// All resident blocks that share `counter` (zero at the start of the kernel) have arrived
// `target` times in all.  A wait runs out when nobody has shown progress for one to two
// periods.  A block whose wait runs out marks the counter, in the same
// word that the arrivals are counted in: either it finds that all have arrived after
// all, or everybody who comes to this barrier or leaves it later sees the mark.  It also
// sets the error word, so that blocks at other counters stop waiting; they arrive at
// theirs all the same.  False: this block gave up.  Whether any block did at any counter
// is known from the error word after the last barrier of all (any_gave_up): read at every
// one it cost 0.6 us each.
__device__ __forceinline__ bool grid_barrier(unsigned* counter, unsigned target, unsigned* error,
                                             const unsigned* progress,
                                             unsigned long long period_ns) {
  __shared__ bool ok, looked;           // (the last two: of a wait that runs long)
  __shared__ unsigned shown;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    atomicAdd(counter, 1u);      // (without its result: the first look is under way at once)
    unsigned seen;
    looked = false;
    while (true) {
      seen = *(volatile unsigned*)counter;
      if (seen >= target) break;            // (a mark is above every target)
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t - t0 > period_ns) {
        const unsigned now = *(const volatile unsigned*)progress;
        if (!looked || now != shown) {
          looked = true;
          shown = now;
          t0 = t;
          continue;
        }
        seen = atomicOr(counter, kGaveUp);
        break;
      }
      if (*(volatile unsigned*)error != 0u) break;
    }
    ok = seen >= target && !(seen & kGaveUp);
    if (!ok) *(volatile unsigned*)error = 1u;
    __threadfence();
  }
  __syncthreads();
  return ok;
}

__device__ __forceinline__ bool any_gave_up(const unsigned* error) {
  return *(const volatile unsigned*)error != 0u;
}

}  // namespace tfgpc
