// Barrier of a cooperative grid for the kernels that run a whole loop (time
// steps, CG iterations) of a small body in one launch.
#pragma once

#include <cuda_runtime.h>

#include "pd_internal.cuh"

namespace pdb {

// Polls of one wait (each a round trip to L2, about a second in all). After
// that the kernel sets ST_TIMEOUT and every block leaves.
constexpr unsigned kGridSpin = 1u << 20;

// bar: [0] blocks arrived, [1] barriers passed, both zero at launch. Writes of
// all blocks before it are visible to all blocks after it. False when the wait
// ran out (in every thread of the block); the caller returns.
__device__ __forceinline__ bool grid_sync(unsigned int* bar, int* status) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int gen, old, cur;
    int good = 1;
    __threadfence();
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(gen) : "l"(bar + 1) : "memory");
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(bar) : "memory");
    if (old == gridDim.x - 1) {
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(bar), "r"(0u) : "memory");
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar + 1) : "memory");
    } else {
      for (unsigned it = 0;; ++it) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(bar + 1) : "memory");
        if (cur != gen) break;
        if (it >= kGridSpin) {
          atomicOr(status, ST_TIMEOUT);
          good = 0;
          break;
        }
      }
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

}  // namespace pdb
