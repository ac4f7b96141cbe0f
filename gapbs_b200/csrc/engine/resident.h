// resident.h -- a single-column gather solve as one cooperative launch
// (resident.cu), and the row tasks its warps take.
#ifndef GAPBS_B200_ENGINE_RESIDENT_H_
#define GAPBS_B200_ENGINE_RESIDENT_H_

#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

namespace prgpu {

constexpr int kResidentThreads = 1024;
// Fewer CTAs on small graphs: one per so many entries, or vertices where those
// are more (1024 vertices, us a solve: 88 with 20 CTAs, 96 with 5, 137 with
// one; 2^24 vertices and 3,000 edges, ms: 6.9 with 5 CTAs, 0.32 with 148).
constexpr int64_t kResidentEntriesPerCta = 1024;

// Polls of a grid barrier before a CTA gives up (about 10 s), on small graphs.
constexpr unsigned kMaxPolls = 1u << 24;

// State of a barrier between a launch's CTAs (grid_barrier.cuh), zero between
// launches; a launch whose wait ran out leaves it to be cleared.
struct GridBarrier {
  unsigned arrived;  // CTAs that arrived, all rounds of a launch together
  unsigned left;     // CTAs that left the launch
};

// Cooperative launch of fn(args) on `grid` CTAs, or on fewer where the stream
// may use part of the GPU only (the kernels take any grid size).
cudaError_t LaunchGrid(const void *fn, int grid, int threads, void *args, size_t smem,
                       cudaStream_t s);

// What a solve tells the host (page-locked host memory).
struct ResidentResult {
  int sweeps;
  int failed;       // a barrier wait ran out
  double sweep_ns;  // device time of the sweeps
};

struct ResidentArgs {
  int32_t n, max_iters;
  const int32_t *__restrict__ rowoff;  // rows to gather
  const int32_t *__restrict__ col;
  const float *__restrict__ win;       // nullable
  const int32_t *__restrict__ odeg;    // directed, unweighted: out-degrees
  const float *__restrict__ rsum;      // weighted: sums of out-weights
  const int32_t *__restrict__ perm;
  const int32_t *__restrict__ inv;
  const float *in_old;  // teleport (adjoint: loss weights), original ids; nullable
  float *out_old;       // scores ((1-d) lambda), original ids; nullable
  float init_scalar, base_scalar, damping, one_minus_d;
  float *score, *c0, *c1, *base;
  // tasks (RowTasks)
  int32_t row_start[kNumBins + 1], task_start[kNumBins + 1];
  const int32_t *__restrict__ order;
  const int4 *__restrict__ seg;
  float *seg_partial;
  unsigned *ticket;
  int32_t segment;           // entries of a long row's segment
  int32_t tile;              // contribs [0, tile) are gathered from shared memory
  int32_t zero_final_sweep;  // from this sweep on rows without entries are final
  double epsilon;
  double *part;   // 2 x CTAs
  double *trace;  // max_iters
  GridBarrier *ctl;
  unsigned max_polls;
  ResidentResult *res;
};

const void *ResidentKernel(int kind, bool weighted, bool directed);

// Lengths that divide the rows: segment (rows of at least as many entries
// are cut into segments), then the shortest row of 32, 16, 8, 4 and 2 lanes.
struct RowClasses {
  int32_t segment;
  int32_t min_len[5];
};
RowClasses ClassesFor(int64_t m, bool weighted);

// Row tasks of a CSR; sorted: its rows already have descending lengths.
cudaError_t BuildRowTasks(int32_t n, const int32_t *rowoff, bool sorted, const RowClasses &rc,
                          RowTasks *r, cudaStream_t s);

}  // namespace prgpu

#endif  // GAPBS_B200_ENGINE_RESIDENT_H_
