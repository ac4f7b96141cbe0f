// grid_barrier.cuh -- a barrier between the CTAs of a cooperative launch.
#ifndef GAPBS_B200_ENGINE_GRID_BARRIER_CUH_
#define GAPBS_B200_ENGINE_GRID_BARRIER_CUH_

#include <cuda_runtime.h>

#include "barrier_count.h"
#include "resident.h"

namespace prgpu {

// polls of the barrier before a CTA gives up (about 10 s)
constexpr unsigned kMaxPolls = 1u << 24;

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Thread 0 of every CTA arrives and waits until all have arrived `round`
// times (1, 2, ... over a launch); false when the wait ran out.  Called by
// all threads; what any CTA wrote before it is visible after it to loads that
// the compiler may not serve from the read-only path.
__device__ __forceinline__ bool grid_barrier(GridBarrier *b, unsigned round, int *s_ok) {
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&b->arrived, 1u);
    const unsigned want = round * gridDim.x;
    unsigned polls = 0;
    while (!arrivals_reached(ld_acquire(&b->arrived), want) && ++polls < kMaxPolls) {
    }
    *s_ok = polls < kMaxPolls;
    __threadfence();
  }
  __syncthreads();
  return *s_ok != 0;
}

// Called by all threads after their last barrier: the last CTA to leave makes
// the barrier ready for the next launch (all have passed their last wait).
__device__ __forceinline__ void leave_grid(GridBarrier *b) {
  if (threadIdx.x != 0) return;
  const unsigned left = atomicAdd(&b->left, 1u);
  if (left == gridDim.x - 1) {
    b->arrived = 0;
    b->left = 0;
  }
}

}  // namespace prgpu

#endif  // GAPBS_B200_ENGINE_GRID_BARRIER_CUH_
