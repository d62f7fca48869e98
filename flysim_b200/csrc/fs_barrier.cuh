// Bounded grid barrier of the persistent kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace fsd {

// ---- bounded grid barrier ---------------------------------------------------
// Over the `count` blocks that share `bar` (the whole grid).  The first 8
// bytes of bar are a 64-bit arrival counter that the host zeroes before each
// launch and that only grows: barrier k of a launch is passed when the
// counter reaches k * count.  Each block's thread 0, after bar.sync (which
// orders the block's writes before it), adds its arrival with a release
// reduction and polls the counter with acquire loads; a load that sees the
// full count synchronises with every arrival (the reductions form one
// release sequence), and the closing bar.sync hands that on to the block.
// No block resets anything and there is no second hop through a
// generation word.  Every wait is bounded: after ~2^24 polls the block sets
// the error word and all blocks leave.  `target` is thread 0's count of the
// arrivals expected so far.
__device__ __forceinline__ unsigned long long ld_acquire_gpu(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu(unsigned long long *p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ bool arrive_and_wait(unsigned int *bar, int *err, uint32_t count,
                                                unsigned long long &target, unsigned int limit) {
  unsigned long long *ctr = (unsigned long long *)bar;
  target += count;
  red_release_gpu(ctr, 1ull);
  // the error word is looked at every 64 polls only: a load after an acquire
  // load waits for it, so checking it on every poll would double the time
  // between polls
  unsigned int spins = 0;
  while (ld_acquire_gpu(ctr) < target) {
    if ((++spins & 63u) == 0u) {
      if (*(volatile int *)err) return false;
      if (spins > limit) {
        atomicExch(err, 2);
        return false;
      }
    }
  }
  return true;
}

// A block leaves when thread 0's wait failed (its own limit, or the error
// word set by another block); thread 0 hands the outcome to the block
// through shared memory, so no thread reads global memory after the
// barrier.  A block that passed a barrier which another block gave up on
// finds the error word set while it waits at the next one (that block never
// arrives there), so every block leaves within 64 polls of the failure.
__device__ __forceinline__ bool grid_sync(unsigned int *bar, int *err, uint32_t count, unsigned long long &target,
                                          unsigned int limit = 1u << 24) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) ok = count > 1 ? arrive_and_wait(bar, err, count, target, limit) : 1;
  __syncthreads();
  return ok != 0;
}

}  // namespace fsd
