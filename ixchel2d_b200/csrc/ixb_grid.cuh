// ixb_grid.cuh -- the barrier of all CTAs of a cooperative launch.
#pragma once
#include <cuda_runtime.h>

namespace ixb {

// All CTAs of the grid: everything written before it (by any thread) is
// visible after it.  The wait is bounded like the other waits of the library
// (polls and about two seconds); false: it ran out, or another CTA gave up.
__device__ __forceinline__ bool grid_sync(unsigned* bar, int* abort_flag, unsigned& target) {
  __shared__ int ok_s;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    bool ok = false;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (int i = 0; i < (1 << 24); ++i) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - target) >= 0) { ok = true; break; }
      if ((i & 1023) == 1023) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > 2000000000ull || *(volatile int*)abort_flag) break;
      }
    }
    if (!ok) *(volatile int*)abort_flag = 1;
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

}  // namespace ixb
