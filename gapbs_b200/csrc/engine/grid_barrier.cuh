// grid_barrier.cuh -- a barrier between the CTAs of a cooperative launch.
#ifndef GAPBS_B200_ENGINE_GRID_BARRIER_CUH_
#define GAPBS_B200_ENGINE_GRID_BARRIER_CUH_

#include <cuda_runtime.h>

#include "barrier_count.h"
#include "resident.h"

namespace prgpu {

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Thread 0 of every CTA arrives and waits until all have arrived `round`
// times (1, 2, ... over a launch); false when the wait ran out after
// max_polls polls.  Called by all threads; what any CTA wrote before it is
// visible after it to loads that the compiler may not serve from the
// read-only path.  A CTA that gives up must return: it arrives no more, so no
// CTA passes the next round, and what one reads after this round is complete.
__device__ __forceinline__ bool grid_barrier(GridBarrier *b, unsigned round, unsigned max_polls,
                                             int *s_ok) {
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&b->arrived, 1u);
    const unsigned want = round * gridDim.x;
    unsigned polls = 0;
    bool all;
    while (!(all = arrivals_reached(ld_acquire(&b->arrived), want)) && polls++ < max_polls) {
    }
    *s_ok = all;
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
