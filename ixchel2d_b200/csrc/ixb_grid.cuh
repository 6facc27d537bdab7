// ixb_grid.cuh -- the waits of all CTAs of a cooperative launch for one another.
#pragma once
#include <cuda_runtime.h>

#include "ixb_grid.h"

namespace ixb {

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(unsigned* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// Start of a resident kernel.  Every CTA reports as it starts (grid_arrive)
// and waits for the others before it writes anything (grid_meet), so that
// what a launch found is whole if its CTAs do not all get an SM: then none of
// them goes on, and the host runs the call another way.  (A cooperative
// launch promises that they do; a GPU shared with long kernels, or a smaller
// partition of one, is where the promise would be missed.)  The outcome is
// the same for all: the word's top bit closes it, and is only set in place
// of a count that is not full.  A launch behind one that gave up does not
// meet either.
__device__ __forceinline__ void grid_arrive(const GridWaits& g) {
  if (threadIdx.x == 0) add_release(&g.words->met);
}
// How long a CTA waits for the last one to start: 0.2 s, beyond which the
// per-sweep kernels get on with the GPU as it is.
__device__ __forceinline__ bool grid_meet(const GridWaits& g) {
  __shared__ int met_s;
  if (threadIdx.x == 0) {
    constexpr unsigned kClosed = 1u << 31;
    const unsigned want = gridDim.x + (g.expire == GRID_EXPIRE_MEET ? 1u : 0u);
    const int polls = g.expire == GRID_EXPIRE_MEET ? 256 : 1 << 24;
    const unsigned long long t0 = global_ns();
    bool met = false;
    const bool over = *(volatile int*)&g.words->gave_up != 0;
    for (int i = 0; !over; ++i) {
      const unsigned v = load_acquire(&g.words->met);
      if (v & kClosed) break;
      if (v >= want) { met = true; break; }
      if (i >= polls || ((i & 255) == 255 && global_ns() - t0 > 200000000ull)) {
        if (atomicCAS(&g.words->met, v, v | kClosed) == v) break;  // else: one more has started
      }
    }
    if (!met && !over) *(volatile int*)&g.words->gave_up = GRID_NOT_MET;
    met_s = met;
  }
  __syncthreads();
  return met_s != 0;
}

// All CTAs of the grid: everything written before it (by any thread) is
// visible after it.  The wait is bounded like the other waits of the library
// (polls and about two seconds); false: it ran out, or another CTA gave up.
__device__ __forceinline__ bool grid_sync(const GridWaits& g, unsigned& target) {
  __shared__ int ok_s;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned want = target + (g.expire == GRID_EXPIRE_SYNC ? 1u : 0u);
    const int polls = g.expire == GRID_EXPIRE_SYNC ? 4096 : 1 << 24;
    add_release(&g.words->bar);
    bool ok = false;
    const unsigned long long t0 = global_ns();
    for (int i = 0; i < polls; ++i) {
      if ((int)(load_acquire(&g.words->bar) - want) >= 0) { ok = true; break; }
      if ((i & 1023) == 1023 && (global_ns() - t0 > 2000000000ull || *(volatile int*)&g.words->gave_up)) break;
    }
    if (!ok) *(volatile int*)&g.words->gave_up = GRID_GAVE_UP;
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

}  // namespace ixb
