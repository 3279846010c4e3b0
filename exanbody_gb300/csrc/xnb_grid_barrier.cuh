// Grid barrier of the cooperative kernels (the persistent step loop and the
// fused rebin), every wait bounded by the global timer.
#pragma once

#include "xnb_internal.cuh"

namespace xnb {

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Blocks count in; the last one resets the count and bumps the generation, the
// others poll the generation for at most wait_ns. A wait that runs out records
// the error and returns false (the kernel then ends without another barrier).
// Once the error is set every later barrier fails at once.
__device__ __forceinline__ bool grid_barrier(GridBarrier* bar, unsigned int nblocks,
                                             unsigned long long wait_ns = 4000000000ull) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    const unsigned int gen = ld_acquire_u32(&bar->generation);
    __threadfence();
    if (ld_acquire_u32(&bar->error)) {
      ok = 0;
    } else if (atomicAdd(&bar->arrive, 1u) == nblocks - 1u) {
      atomicExch(&bar->arrive, 0u);
      __threadfence();
      atomicAdd(&bar->generation, 1u);
    } else {
      const unsigned long long t0 = global_ns();
      while (ld_acquire_u32(&bar->generation) == gen) {
        if (global_ns() - t0 > wait_ns) {
          atomicOr(&bar->error, 1u);
          ok = 0;
          break;
        }
        __nanosleep(40);
      }
    }
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}

}  // namespace xnb
