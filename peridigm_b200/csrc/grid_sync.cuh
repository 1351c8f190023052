// Barrier of a cooperative grid for the kernels that run a whole loop (time
// steps, CG iterations) of a small body in one launch.
#pragma once

#include <cuda_runtime.h>

#include "pd_internal.cuh"

namespace pdb {

// Polls of one wait (each a round trip to L2, about a second in all). After
// that the block sets ST_TIMEOUT and leaves, and so do those that wait for it. (A
// constant: with a limit from a kernel argument each barrier took 75 ns more.)
constexpr unsigned kGridSpin = 1u << 20;

// bar: blocks arrived since the launch, zero then; target: of the next barrier,
// zero at the kernel's start. Writes of all blocks before it are visible to all
// blocks after it (release by the block's arrival, acquire by its wait, for
// the whole block through the block barriers). One message out and one poll
// back: an arrival counter that is never reset needs neither the atomic's answer
// nor a second word. False when the wait ran out (in every thread of the
// block); the caller returns.
__device__ __forceinline__ bool grid_sync(unsigned int* bar, unsigned int& target, int* status) {
  __shared__ int ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    int good = 1;
    for (unsigned it = 0;; ++it) {
      unsigned int cur;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(bar) : "memory");
      if ((int)(cur - target) >= 0) break;
      if (it >= kGridSpin) {
        atomicOr(status, ST_TIMEOUT);
        good = 0;
        break;
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

}  // namespace pdb
