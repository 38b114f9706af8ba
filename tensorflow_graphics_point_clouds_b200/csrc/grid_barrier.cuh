// Barrier over blocks of a cooperative launch, with a bounded wait.
#pragma once

#include "common.cuh"

namespace tfgpc {

constexpr unsigned kGaveUp = 0x80000000u;    // in a barrier's counter

// All resident blocks that share `counter` (zero at the start of the kernel) have arrived
// `target` times in all.  A block whose wait runs out marks the counter, in the same
// word that the arrivals are counted in: either it finds that all have arrived after
// all, or everybody who comes to this barrier or leaves it later sees the mark.  It also
// sets the error word, so that blocks at other counters stop waiting; they arrive at
// theirs all the same.  False: this block gave up.  Whether any block did at any counter
// is known from the error word after the last barrier of all (any_gave_up): read at every
// one it cost 0.6 us each.
__device__ __forceinline__ bool grid_barrier(unsigned* counter, unsigned target, unsigned* error,
                                             unsigned long long limit_ns) {
  __shared__ bool ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    atomicAdd(counter, 1u);      // (without its result: the first look is under way at once)
    unsigned seen;
    while (true) {
      seen = *(volatile unsigned*)counter;
      if (seen >= target) break;            // (a mark is above every target)
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t - t0 > limit_ns) {
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
