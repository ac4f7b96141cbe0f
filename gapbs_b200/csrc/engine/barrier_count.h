// barrier_count.h -- the count a grid barrier waits for (grid_barrier.cuh);
// plain C++, so that the host can check it.
#ifndef GAPBS_B200_ENGINE_BARRIER_COUNT_H_
#define GAPBS_B200_ENGINE_BARRIER_COUNT_H_

#ifdef __CUDACC__
#define PR_HOST_DEVICE __host__ __device__
#else
#define PR_HOST_DEVICE
#endif

namespace prgpu {

// Whether the count of a launch's arrivals has reached `want` = round x CTAs.
// Both are kept modulo 2^32 (296 CTAs pass it after 14.5 M rounds, and a
// search of a long chain takes a round per vertex).  No CTA is more than a
// round ahead of another, so the two differ by less than 2^31.
PR_HOST_DEVICE constexpr bool arrivals_reached(unsigned arrived, unsigned want) {
  return static_cast<int>(arrived - want) >= 0;
}

}  // namespace prgpu

#endif  // GAPBS_B200_ENGINE_BARRIER_COUNT_H_
