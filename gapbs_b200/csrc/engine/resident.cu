// resident.cu -- a whole single-column gather solve in one launch.
//
// The replaced code is src/pr_spmv.cc:37-60: init, sweeps of
//   sum   = sum over in-neighbours v of contrib[v]
//   new   = base + d * sum                      (float, two roundings)
//   err  += |new - old|                          (float difference, FP64 sum)
//   contrib'[u] = new / out_degree(u)            (next sweep's input)
// until err < epsilon, and the scores in the caller's order; the same for
// personalized PageRank (base a vector) and the adjoint iteration (out-rows,
// the gathered value is the new value itself).
//
// One 1024-thread CTA per SM stays for the whole solve (cooperative launch,
// so all of them are resident) and the sweeps are separated by a grid
// barrier.  Two things bound a gather sweep and are taken out of its way:
//   * an SM serves one 128-byte line of L1 or L2 per clock to a scattered
//     load (148 SMs: 285 G gathers/s, measured), whether the line hits L1 or
//     not.  Shared memory serves 32 banks per clock, so the contribs of the
//     first `tile` vertices -- the highest in-degrees, which most edges come
//     from -- are copied into shared memory at the start of each sweep and
//     gathered there;
//   * a launch per sweep costs ~10 us between dependent sweeps of a
//     conditional graph, the barrier ~2 us.
//
// Work split: rows in descending-length order (the in-rows are renumbered
// so; out-rows of directed graphs come through `order`).  Rows of at least
// `segment` entries are cut into segments of as many entries, one warp each;
// the warp that brings a row's last segment (per-row ticket) sums the row's
// partials by a fixed tree.  Shorter rows go to groups of 32 .. 1 lanes by
// length, two rows a lane group at once below 32 lanes, rows without entries
// to plain lanes.  Tasks are dealt to the warps of the grid in a fixed order,
// neighbours to different SMs: every sum has a fixed tree, so a solve's bits
// do not depend on timing.
//
// Every wait on the barrier is bounded: a CTA that gives up sets the error
// flag and returns, and so do the others when their own waits run out.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "grid_barrier.cuh"
#include "resident.h"

namespace prgpu {

namespace {

constexpr int kThreads = kResidentThreads;
constexpr int kWarps = kThreads / 32;
static_assert(kWarps == 32, "one warp sums the warps' partials");
constexpr unsigned kFull = 0xffffffffu;
// Entry v of cin: from shared memory below `tile`, else from L2 (other CTAs
// wrote it in the sweep before, and L1 is not coherent within a launch).
// v == -1 reads the zero slot in front of the tile.  Both loads are predicated,
// so a warp whose lanes need both issues two instructions and no branch.
__device__ __forceinline__ float gather1(unsigned tile_sm, int tile, const float *cin, int v,
                                         uint64_t pol) {
  float r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.lt.s32 p, %1, %2;\n\t"
      "@p ld.shared.f32 %0, [%3];\n\t"
      "@!p ld.global.cg.L2::cache_hint.f32 %0, [%4], %5;\n\t}"
      : "=f"(r)
      : "r"(v), "r"(tile), "r"(tile_sm + (static_cast<unsigned>(v) << 2)), "l"(cin + v), "l"(pol));
  return r;
}

__device__ __forceinline__ void cp_async_16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Sum of the CTAs' partials in a fixed order, by one warp; valid in lane 0.
__device__ __forceinline__ double sum_partials(const double *part, int lane) {
  double v = 0;
  for (int i = lane; i < static_cast<int>(gridDim.x); i += 32) v += __ldcg(part + i);
  return warp_sum_d(v);
}

template <bool W, bool DIR>
__device__ __forceinline__ float denom(const ResidentArgs &a, int u, int s, int e) {
  if (W) return a.rsum[u];
  if (DIR) return __int2float_rn(a.odeg[u]);
  return __int2float_rn(e - s);
}

// One lane's share of a row: entries [s, e) in aligned four-entry chunks
// c, c + step, ...  A graph may have 2^31 - 9 entries, so the first entry of a
// chunk past the row's end needs all 32 bits: unsigned.
struct Share {
  int s, e, c;
  __device__ __forceinline__ unsigned first() const { return static_cast<unsigned>(c) << 2; }
  __device__ __forceinline__ bool more() const { return first() < static_cast<unsigned>(e); }
};

template <bool W>
__device__ __forceinline__ void load_chunk(const ResidentArgs &a, const Share &x, int4 &q,
                                           float4 &w, uint64_t ps) {
  if (!x.more()) return;
  q = ld_stream_v4(reinterpret_cast<const int4 *>(a.col) + x.c, ps);
  if (W) w = ld_stream_v4f(reinterpret_cast<const float4 *>(a.win) + x.c, ps);
}

// Adds chunk x.c; entries outside the row become the id of the zero slot.
template <bool W>
__device__ __forceinline__ void add_chunk(float &acc, const Share &x, const int4 &q,
                                          const float4 &w, const float *cin, unsigned tile_sm,
                                          int tile, uint64_t pg) {
  if (!x.more()) return;
  const unsigned len = x.e - x.s;
  const unsigned d = x.first() - x.s;  // wraps below the row's start
  const float v0 = gather1(tile_sm, tile, cin, d < len ? q.x : -1, pg);
  const float v1 = gather1(tile_sm, tile, cin, d + 1 < len ? q.y : -1, pg);
  const float v2 = gather1(tile_sm, tile, cin, d + 2 < len ? q.z : -1, pg);
  const float v3 = gather1(tile_sm, tile, cin, d + 3 < len ? q.w : -1, pg);
  if (W) {
    acc = __fmaf_rn(w.x, v0, acc);
    acc = __fmaf_rn(w.y, v1, acc);
    acc = __fmaf_rn(w.z, v2, acc);
    acc = __fmaf_rn(w.w, v3, acc);
  } else {
    acc = __fadd_rn(acc, __fadd_rn(__fadd_rn(v0, v1), __fadd_rn(v2, v3)));
  }
}

// Two shares at once, so that the chunk loads and gathers of both are in
// flight together.
template <bool W>
__device__ __forceinline__ void sum_shares(const ResidentArgs &a, Share x, Share y, int step,
                                           const float *cin, unsigned tile_sm, uint64_t ps,
                                           uint64_t pg, float &acc_x, float &acc_y) {
  acc_x = acc_y = 0.f;
  while (x.more() || y.more()) {
    int4 qx, qy;
    float4 wx, wy;
    load_chunk<W>(a, x, qx, wx, ps);
    load_chunk<W>(a, y, qy, wy, ps);
    add_chunk<W>(acc_x, x, qx, wx, cin, tile_sm, a.tile, pg);
    add_chunk<W>(acc_y, y, qy, wy, cin, tile_sm, a.tile, pg);
    x.c += step;
    y.c += step;
  }
}

// Row u from its gathered sum; returns |new - old|.
template <bool W, bool DIR, int KIND>
__device__ __forceinline__ float finish_row(const ResidentArgs &a, float *cout, int u, int s,
                                            int e, float sum, float old, uint64_t ps,
                                            uint64_t pl) {
  const float base = KIND != kKindPlain ? a.base[u] : a.base_scalar;
  const float den = denom<W, DIR>(a, u, s, e);
  float nw, out;
  if (KIND == kKindAdjoint) {
    // a vertex without out-edges has no row in P: (P lambda)[v] = 0
    const float p = den > 0.f ? __fdiv_rn(sum, den) : 0.f;
    nw = __fadd_rn(base, __fmul_rn(a.damping, p));
    out = nw;
  } else {
    nw = __fadd_rn(base, __fmul_rn(a.damping, sum));
    out = __fdiv_rn(nw, den);
  }
  st_hint_f32(a.score + u, nw, ps);
  st_hint_f32(cout + u, out, pl);
  return fabsf(__fsub_rn(nw, old));
}

// What one lane takes of a task: two rows of a lane group of 2^lg lanes
// (bins 2 .. 6), or one row or segment (second == u, lg = 5).
struct Task {
  int u, s, e;
  int u2, s2, e2;
  int lg;
};

// Row positions past a bin's end (up to 511 of them) may pass 2^31: unsigned.
__device__ __forceinline__ Task load_task(const ResidentArgs &a, int t, int ntasks, int lane32) {
  Task x{0, 0, 0, 0, 0, 0, 5};
  if (t >= min(ntasks, a.task_start[kBinZero])) return x;
  if (t < a.task_start[1]) {
    const int4 sg = a.seg[t];
    x.u = sg.x;
    x.s = sg.z;
    x.e = sg.w;
    return x;
  }
  int bin = 1;
#pragma unroll
  for (int i = 2; i < kBinZero; i++) bin += (t >= a.task_start[i]);
  x.lg = 6 - bin;  // 32, 16, 8, 4, 2, 1 lanes a row
  const int k = (t - a.task_start[bin]) << (bin > 1 ? 6 - x.lg : 0);
  const unsigned p = static_cast<unsigned>(a.row_start[bin]) + k + (lane32 >> x.lg);
  const unsigned end = a.row_start[bin + 1];
  if (p < end) {
    x.u = a.order ? a.order[p] : p;
    x.s = a.rowoff[x.u];
    x.e = a.rowoff[x.u + 1];
  }
  const unsigned p2 = p + (32 >> x.lg);
  if (bin > 1 && p2 < end) {
    x.u2 = a.order ? a.order[p2] : p2;
    x.s2 = a.rowoff[x.u2];
    x.e2 = a.rowoff[x.u2 + 1];
  }
  return x;
}

template <bool W, bool DIR, int KIND>
__global__ void __launch_bounds__(kThreads, 1) resident_solve_kernel(const ResidentArgs a) {
  // four words of which the last is the zero slot, then the tile
  extern __shared__ __align__(16) float sm[];
  __shared__ double s_red[kWarps];
  __shared__ double s_tot;
  __shared__ int s_ok;
  const uint64_t ps = policy_evict_first();
  const uint64_t pl = policy_evict_last();
  const int lane32 = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned tile_sm = static_cast<unsigned>(__cvta_generic_to_shared(sm + 4));
  unsigned round = 0;
  const int64_t gthreads = static_cast<int64_t>(gridDim.x) * kThreads;
  const int64_t gtid = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;

  // ---- init: s_0 = t (1/N), base = (1-d) t, contrib = s_0 / out_degree;
  // adjoint: lambda_0 = base = w, and ||w||_1 for the stop rule
  double norm = 0;
  for (int64_t i = gtid; i < a.n; i += gthreads) {
    const int u = static_cast<int>(i);
    const float t = a.in_old ? a.in_old[a.perm[u]] : a.init_scalar;
    a.score[u] = t;
    if (KIND == kKindAdjoint) {
      a.base[u] = t;
      a.c0[u] = t;
      norm += static_cast<double>(fabsf(t));
    } else {
      if (KIND == kKindPPR) a.base[u] = __fmul_rn(a.one_minus_d, t);
      a.c0[u] = __fdiv_rn(t, denom<W, DIR>(a, u, W || DIR ? 0 : a.rowoff[u],
                                           W || DIR ? 0 : a.rowoff[u + 1]));
    }
  }
  if (threadIdx.x == 0) sm[3] = 0.f;
  double epsilon = a.epsilon;
  if (KIND == kKindAdjoint) {
    norm = warp_sum_d(norm);
    if (lane32 == 0) s_red[wid] = norm;
    __syncthreads();
    if (wid == 0) {
      const double v = warp_sum_d(s_red[lane32]);
      if (lane32 == 0) a.part[gridDim.x + blockIdx.x] = v;  // the slot of odd sweeps
    }
  }
  if (!grid_barrier(a.ctl, ++round, a.max_polls, &s_ok)) {
    if (threadIdx.x == 0) a.res->failed = 1;
    return;
  }
  if (KIND == kKindAdjoint) {
    if (wid == 0) {
      const double t = sum_partials(a.part + gridDim.x, lane32);
      if (lane32 == 0) s_tot = t;
    }
    __syncthreads();
    epsilon *= s_tot;
  }
  unsigned long long t_begin = 0;
  if (gtid == 0) t_begin = global_ns();

  // ---- sweeps
  const int gw = wid * gridDim.x + blockIdx.x;
  const int nw = gridDim.x * kWarps;
  int it = 0;
  for (; it < a.max_iters; it++) {
    const float *cin = (it & 1) ? a.c1 : a.c0;
    float *cout = (it & 1) ? a.c0 : a.c1;
    double *part = a.part + (it & 1 ? gridDim.x : 0);
    for (int i = threadIdx.x; i < (a.tile >> 2); i += kThreads)
      cp_async_16(tile_sm + 16u * i, cin + 4 * i);
    cp_async_wait_all();
    __syncthreads();
    double err = 0;  // every |new - old| added in FP64 (src/pr_spmv.cc:42,53)
    const int ntasks = it >= a.zero_final_sweep ? a.task_start[kBinZero] : a.task_start[kNumBins];
    // tasks in descending size are dealt back and forth, which evens out the
    // warps' sums; the bounds of a warp's next task are fetched before the
    // current one is gathered
    Task x = load_task(a, gw, ntasks, lane32);
    int t = gw, back = nw - 1 - 2 * gw;  // from a round's place to its mirror image
    while (t < a.task_start[kBinZero]) {
      const int tn = t + nw + back;
      back = -back;
      const Task y = load_task(a, tn, ntasks, lane32);
      const bool one_row = x.lg == 5;  // both shares are of the one row
      const int lane = lane32 & ((1 << x.lg) - 1);
      Share p{x.s, x.e, (x.s >> 2) + lane};
      Share q{x.s2, x.e2, (x.s2 >> 2) + lane};
      if (one_row) q = Share{x.s, x.e, p.c + 32};
      const bool segment = t < a.task_start[1];
      float old = 0.f, old2 = 0.f;
      if (lane == 0 && !segment) {
        if (x.e > x.s) old = __ldcg(a.score + x.u);
        if (x.e2 > x.s2) old2 = __ldcg(a.score + x.u2);
      }
      float acc, acc2;
      sum_shares<W>(a, p, q, one_row ? 64 : 1 << x.lg, cin, tile_sm, ps, pl, acc, acc2);
      if (one_row) acc += acc2;
      for (int o = (1 << x.lg) >> 1; o > 0; o >>= 1) {
        acc += __shfl_xor_sync(kFull, acc, o);
        acc2 += __shfl_xor_sync(kFull, acc2, o);
      }
      if (lane == 0) {
        if (segment) {
          a.seg_partial[t] = acc;
        } else {
          if (x.e > x.s) err += finish_row<W, DIR, KIND>(a, cout, x.u, x.s, x.e, acc, old, ps, pl);
          if (x.e2 > x.s2)
            err += finish_row<W, DIR, KIND>(a, cout, x.u2, x.s2, x.e2, acc2, old2, ps, pl);
        }
      }
      x = y;
      t = tn;
    }
    // rows without entries: new = base
    for (; t < ntasks; t += nw + back, back = -back) {
      const unsigned p0 = static_cast<unsigned>(a.row_start[kBinZero]) +
                          (t - a.task_start[kBinZero]) * (32 * kZeroRowsPerThread) + lane32;
#pragma unroll
      for (int i = 0; i < kZeroRowsPerThread; i++) {
        const unsigned p = p0 + 32 * i;
        if (p < static_cast<unsigned>(a.n)) {
          const int u = a.order ? a.order[p] : p;
          err += finish_row<W, DIR, KIND>(a, cout, u, 0, 0, 0.f, __ldcg(a.score + u), ps, pl);
        }
      }
    }
    // long rows: the warp that brings a row's last segment finishes the row
    // (one fence a warp and sweep: a fence per segment stalled the warps)
    if (gw < a.task_start[1]) {
      __threadfence();
      back = nw - 1 - 2 * gw;
      for (int k = gw; k < a.task_start[1]; k += nw + back, back = -back) {
        const int4 sg = a.seg[k];
        const int rs = a.rowoff[sg.x], re = a.rowoff[sg.x + 1];
        const int nseg = static_cast<int>((static_cast<unsigned>(re - rs) + a.segment - 1u) /
                                          static_cast<unsigned>(a.segment));
        int last = 0;
        if (lane32 == 0)
          last = atomicAdd(a.ticket + sg.y, 1u) == static_cast<unsigned>(nseg - 1);
        if (!__shfl_sync(kFull, last, 0)) continue;
        __threadfence();
        float sum = 0.f;
        for (int j = lane32; j < nseg; j += 32) sum += __ldcg(a.seg_partial + sg.y + j);
        sum = warp_sum_f(sum);
        if (lane32 == 0) {
          a.ticket[sg.y] = 0;
          err += finish_row<W, DIR, KIND>(a, cout, sg.x, rs, re, sum, __ldcg(a.score + sg.x), ps,
                                          pl);
        }
      }
    }
    err = warp_sum_d(err);
    if (lane32 == 0) s_red[wid] = err;
    __syncthreads();
    if (wid == 0) {
      const double v = warp_sum_d(s_red[lane32]);
      if (lane32 == 0) part[blockIdx.x] = v;
    }
    if (!grid_barrier(a.ctl, ++round, a.max_polls, &s_ok)) {
      if (threadIdx.x == 0) a.res->failed = 1;
      return;
    }
    if (wid == 0) {
      const double t = sum_partials(part, lane32);
      if (lane32 == 0) s_tot = t;
    }
    __syncthreads();
    const double tot = s_tot;
    if (gtid == 0) a.trace[it] = tot;
    if (tot < epsilon) {
      it++;
      break;
    }
  }

  // ---- the scores (adjoint: (1-d) lambda) in the caller's order
  if (gtid == 0) {
    a.res->sweeps = it;
    a.res->sweep_ns = static_cast<double>(global_ns() - t_begin);
  }
  if (a.out_old) {
    for (int64_t v = gtid; v < a.n; v += gthreads) {
      const float x = __ldcg(a.score + a.inv[v]);
      a.out_old[v] = KIND == kKindAdjoint ? __fmul_rn(a.one_minus_d, x) : x;
    }
  }
  leave_grid(a.ctl);
}

template <bool W, bool DIR>
const void *ForKind(int kind) {
  if (kind == kKindPlain)
    return reinterpret_cast<const void *>(resident_solve_kernel<W, DIR, kKindPlain>);
  if (kind == kKindPPR)
    return reinterpret_cast<const void *>(resident_solve_kernel<W, DIR, kKindPPR>);
  return reinterpret_cast<const void *>(resident_solve_kernel<W, DIR, kKindAdjoint>);
}

// First row position of each bin: rows in `order` (or as they are) have
// descending lengths.
__global__ void row_bounds_kernel(int32_t n, const int32_t *__restrict__ rowoff,
                                  const int32_t *__restrict__ order, BinConfig cfg,
                                  int32_t *start) {
  const int b = threadIdx.x;
  if (b > kNumBins) return;
  if (b == 0 || b == kNumBins) {
    start[b] = b ? n : 0;
    return;
  }
  const int t = cfg.min_len[b - 1];
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = lo + ((hi - lo) >> 1);
    const int u = order ? order[mid] : mid;
    if (rowoff[u + 1] - rowoff[u] >= t) lo = mid + 1; else hi = mid;
  }
  start[b] = lo;
}

__global__ void row_lengths_kernel(int32_t count, const int32_t *__restrict__ rowoff,
                                   int32_t *len) {
  const unsigned u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u < static_cast<unsigned>(count)) len[u] = rowoff[u + 1] - rowoff[u];
}

// (row, first entry, end) of the rows at positions 0 .. count-1.
__global__ void long_rows_kernel(int32_t count, const int32_t *__restrict__ rowoff,
                                 const int32_t *__restrict__ order, int32_t *row) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= count) return;
  const int u = order ? order[p] : p;
  row[3 * p] = u;
  row[3 * p + 1] = rowoff[u];
  row[3 * p + 2] = rowoff[u + 1];
}

__global__ void iota_kernel(int32_t n, int32_t *ids) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < static_cast<unsigned>(n)) ids[i] = static_cast<int32_t>(i);
}

// Positions 0 .. n-1 of rows by descending length (stable).
cudaError_t SortRows(int32_t n, const int32_t *rowoff, int32_t *order, cudaStream_t s) {
  int32_t *len = nullptr, *len_sorted = nullptr, *ids = nullptr;
  void *tmp = nullptr;
  size_t bytes = 0;
  cudaError_t e = cudaMalloc(&len, sizeof(int32_t) * n);
  if (e == cudaSuccess) e = cudaMalloc(&len_sorted, sizeof(int32_t) * n);
  if (e == cudaSuccess) e = cudaMalloc(&ids, sizeof(int32_t) * n);
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, len, len_sorted, ids, order, n,
                                                  0, 32, s);
  if (e == cudaSuccess) e = cudaMalloc(&tmp, bytes);
  if (e == cudaSuccess) {
    const unsigned blocks = (static_cast<unsigned>(n) + 255u) / 256u;
    row_lengths_kernel<<<blocks, 256, 0, s>>>(n, rowoff, len);
    iota_kernel<<<blocks, 256, 0, s>>>(n, ids);
    e = cub::DeviceRadixSort::SortPairsDescending(tmp, bytes, len, len_sorted, ids, order, n, 0,
                                                  32, s);
  }
  const cudaError_t done = cudaStreamSynchronize(s);
  for (void *p : {static_cast<void *>(len), static_cast<void *>(len_sorted),
                  static_cast<void *>(ids), tmp})
    if (p) cudaFree(p);
  return e == cudaSuccess ? done : e;
}

}  // namespace

cudaError_t LaunchGrid(const void *fn, int grid, int threads, void *args, size_t smem,
                       cudaStream_t s) {
  void *params[] = {args};
  for (;; grid /= 2) {
    const cudaError_t e =
        cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), params, smem, s);
    if (e != cudaErrorCooperativeLaunchTooLarge || grid == 1) return e;
    cudaGetLastError();
  }
}

void FreeRowTasks(RowTasks *r) {
  for (void *p : {static_cast<void *>(r->order), static_cast<void *>(r->seg),
                  static_cast<void *>(r->ticket), static_cast<void *>(r->seg_partial)})
    if (p) cudaFree(p);
  *r = RowTasks();
}

// Row classes by the entries a warp of a full grid gets, measured (us a solve
// of 6 to 9 sweeps; fine / medium / coarse):
//   Kronecker 2^13, 2^16 vertices  (46, 380 entries a warp)    112 / 113 / 118, 131 / 128 / 135
//   uniform 2^18, 2^20             (1,800, 7,100)              266 / 270 / 296, 1006 / 919 / 925
//   Kronecker 2^18, 2^20           (1,600, 6,600)              257 / 228 / 201,  733 / 620 / 541
//   weighted 2^20 training step                              14123 / 13042 / 13422
// Few entries: small tasks, so that all warps have one.  Many: more entries a
// lane, since each task pays the latency of its chain of loads once.
RowClasses ClassesFor(int64_t m, bool weighted) {
  const int64_t per_warp = m / (148 * kWarps);
  if (per_warp < 256) return RowClasses{1024, {128, 64, 32, 16, 8}};
  if (per_warp < 2048 || weighted) return RowClasses{1024, {256, 128, 64, 32, 16}};
  return RowClasses{2048, {512, 256, 128, 48, 16}};
}

cudaError_t BuildRowTasks(int32_t n, const int32_t *rowoff, bool sorted, const RowClasses &rc,
                          RowTasks *r, cudaStream_t s) {
  FreeRowTasks(r);
  r->segment = rc.segment;
  cudaError_t e = cudaSuccess;
  if (!sorted) {
    e = cudaMalloc(&r->order, sizeof(int32_t) * n);
    if (e == cudaSuccess) e = SortRows(n, rowoff, r->order, s);
  }
  int32_t *d = nullptr;
  if (e == cudaSuccess) e = cudaMalloc(&d, sizeof(int32_t) * (kNumBins + 1));
  if (e == cudaSuccess) {
    BinConfig cfg;
    cfg.min_len[kBinHub] = rc.segment;
    for (int b = 1; b < 6; b++) cfg.min_len[b] = rc.min_len[b - 1];
    row_bounds_kernel<<<1, 32, 0, s>>>(n, rowoff, r->order, cfg, d);
    e = cudaMemcpyAsync(r->row_start, d, sizeof(r->row_start), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (d) cudaFree(d);
  const int32_t nlong = e == cudaSuccess ? r->row_start[1] : 0;
  std::vector<int32_t> row(3 * static_cast<size_t>(nlong));
  if (nlong) {
    e = cudaMalloc(&d, sizeof(int32_t) * row.size());
    if (e == cudaSuccess) {
      long_rows_kernel<<<(nlong + 255) / 256, 256, 0, s>>>(nlong, rowoff, r->order, d);
      e = cudaMemcpyAsync(row.data(), d, sizeof(int32_t) * row.size(), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      cudaFree(d);
    }
  }
  std::vector<int4> seg;
  for (int32_t p = 0; p < nlong && e == cudaSuccess; p++) {
    const int32_t first = static_cast<int32_t>(seg.size());
    const int64_t end = row[3 * p + 2];  // b + segment may pass 2^31
    for (int64_t b = row[3 * p + 1]; b < end; b += rc.segment)
      seg.push_back(make_int4(row[3 * p], first, static_cast<int>(b),
                              static_cast<int>(std::min(end, b + rc.segment))));
  }
  if (e == cudaSuccess && nlong) {
    e = cudaMalloc(&r->seg, sizeof(int4) * seg.size());
    if (e == cudaSuccess) e = cudaMalloc(&r->seg_partial, sizeof(float) * seg.size());
    if (e == cudaSuccess) e = cudaMalloc(&r->ticket, sizeof(unsigned) * seg.size());
    if (e == cudaSuccess) e = cudaMemsetAsync(r->ticket, 0, sizeof(unsigned) * seg.size(), s);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(r->seg, seg.data(), sizeof(int4) * seg.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (e != cudaSuccess) {
    FreeRowTasks(r);
    return e;
  }
  int64_t tasks = static_cast<int64_t>(seg.size());
  r->task_start[0] = 0;
  for (int b = 1; b < kNumBins; b++) {
    r->task_start[b] = static_cast<int32_t>(tasks);
    const int64_t rows = r->row_start[b + 1] - r->row_start[b];
    const int64_t per =
        b == kBinZero ? 32 * kZeroRowsPerThread : (b > 1 ? 2 : 1) * 32 / kBinGroup[b];
    tasks += (rows + per - 1) / per;
  }
  r->task_start[kNumBins] = static_cast<int32_t>(tasks);
  r->ready = true;
  return cudaSuccess;
}

const void *ResidentKernel(int kind, bool weighted, bool directed) {
  if (weighted) return ForKind<true, false>(kind);
  // the adjoint divides by the length of the row it gathers
  if (directed && kind != kKindAdjoint) return ForKind<false, true>(kind);
  return ForKind<false, false>(kind);
}

}  // namespace prgpu
