// verify.cu -- the reference's PRVerifier (src/pr_spmv.cc:78-94) on the device.
//
// The reference pushes contrib[u] = score[u] / out_degree(u) along the
// out-edges of u = 0, 1, 2, ... in turn, so incoming[v] is the float sum of
// v's in-neighbours' contribs in ascending source order, and the check is
// error = sum over n of |base + d * incoming[n] - score[n]| (float
// arithmetic per vertex, added in double in vertex order).
//
// The renumbered in-CSR keeps every row in the caller's order, and the
// reference's builder sorts each row by source id (src/builder.h:154-156), so
// adding a row's contribs one at a time in row order gives incoming[v] bit for
// bit.  Rows are in descending-length order: a block takes each of the longest
// rows, a warp each of the other long ones and a thread each of the short
// ones.  All add a row's terms one after the other, however they are fetched,
// so the sum keeps its sequential rounding.  The residual of each row is
// written at the vertex's original id, and SumInOrder adds them with the
// rounding of the reference's loop over the ids.  Nothing
// here shares code with the sweep kernels, so the check does not inherit a
// fault of theirs.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace prgpu {

namespace {

constexpr int kVerifyThreads = 256;
constexpr int kLongRow = 32;  // rows of at least this many entries get a warp
constexpr int kHubChunk = 1792;  // contribs of a hub row fetched at once by its block
constexpr int kRunLen = 256;     // residuals of a run (SumInOrder)
constexpr unsigned kFull = 0xffffffffu;

// contrib[v] = score[perm[v]] / out_degree(v) over new ids: the float score
// divided by the degree converted to float (src/pr_spmv.cc:83).  A vertex
// without out-edges gets inf or NaN, as in the reference; no row reads it.
__global__ void verify_contrib_kernel(int64_t n, const float *__restrict__ score_orig,
                                      const int32_t *__restrict__ perm,
                                      const int32_t *__restrict__ rowoff,
                                      const int32_t *__restrict__ odeg, float *contrib) {
  const int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const int32_t deg = odeg ? odeg[v] : rowoff[v + 1] - rowoff[v];
  contrib[v] = __fdiv_rn(score_orig[perm[v]], __int2float_rn(deg));
}

// resid_orig[perm[u]] = |base + d * sum - score|, each operation rounded on
// its own (src/pr_spmv.cc:89).
__device__ __forceinline__ void write_residual(int64_t u, float sum,
                                               const float *__restrict__ score_orig,
                                               const int32_t *__restrict__ perm, float base,
                                               float damping, float *resid_orig) {
  const int32_t v = perm[u];
  const float r = __fsub_rn(__fadd_rn(base, __fmul_rn(damping, sum)), score_orig[v]);
  resid_orig[v] = fabsf(r);
}

// The rows, one launch: blocks [0, nhub) take a hub row (at least 4,096
// entries) each, the next blocks a row of at least kLongRow entries per warp,
// the rest a row per thread.  Blocks start in order, so the longest rows,
// which bound the launch, start first.
struct VerifyArgs {
  int64_t n, nhub, nlong;
  unsigned long_blocks;
  const int32_t *__restrict__ rowoff;
  const int32_t *__restrict__ col;
  const float *__restrict__ contrib;
  const float *__restrict__ score_orig;
  const int32_t *__restrict__ perm;
  float base, damping;
  float *resid_orig;
};

__device__ __forceinline__ void residual(const VerifyArgs &a, int64_t u, float sum) {
  write_residual(u, sum, a.score_orig, a.perm, a.base, a.damping, a.resid_orig);
}

// A hub's sum is one chain of dependent float adds (4 cycles each), so the
// block's other warps bring the contribs, kHubChunk at a time, into one of two
// buffers while the first warp adds the other one's in order.  (Fetched by
// the adding warp itself, 32 at a time, the longest row of Kronecker 2^22,
// 163,000 entries, took 3.3 ms of a 3.4 ms launch; the whole is 0.76 ms this
// way.)
__device__ __forceinline__ void hub_row(const VerifyArgs &a, float (*buf)[kHubChunk]) {
  constexpr int kFetchers = kVerifyThreads - 32;
  constexpr int kPer = kHubChunk / kFetchers;
  static_assert(kHubChunk % kFetchers == 0, "whole rounds of fetches");
  const int t = static_cast<int>(threadIdx.x) - 32;  // the first warp never waits for loads
  const int64_t u = blockIdx.x;
  const uint32_t lo = a.rowoff[u], hi = a.rowoff[u + 1];  // at + kHubChunk may pass 2^31
  float v[kPer];
  auto fetch = [&](uint32_t at) {
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      const uint32_t j = at + i * kFetchers + t;
      v[i] = j < hi ? a.contrib[a.col[j]] : 0.f;
    }
  };
  if (t >= 0) fetch(lo);
  float sum = 0.f;
  int k = 0;
  for (uint32_t at = lo; at < hi; at += kHubChunk, k ^= 1) {
    if (t >= 0) {
#pragma unroll
      for (int i = 0; i < kPer; i++) buf[k][i * kFetchers + t] = v[i];
    }
    __syncthreads();  // buffer k is complete; the other one has been added
    if (t >= 0) {
      if (at + kHubChunk < hi) fetch(at + kHubChunk);
    } else {
      const int cnt = min(static_cast<uint32_t>(kHubChunk), hi - at);
      const float4 *b4 = reinterpret_cast<const float4 *>(buf[k]);
      int j = 0;
#pragma unroll 8
      for (; j + 3 < cnt; j += 4) {
        const float4 x = b4[j >> 2];
        sum = __fadd_rn(sum, x.x);
        sum = __fadd_rn(sum, x.y);
        sum = __fadd_rn(sum, x.z);
        sum = __fadd_rn(sum, x.w);
      }
      for (; j < cnt; j++) sum = __fadd_rn(sum, buf[k][j]);
    }
  }
  if (threadIdx.x == 0) residual(a, u, sum);
}

// A warp per row: the row's contribs are fetched 32 at a time, the next 32
// while the current ones are added; every lane keeps the same running sum.
// (32 rows per warp through a transposed shared tile, a lane adding each, took
// a fifth of the instructions but waited for two loads every 8 rows of 32
// entries: 2,900 us for the launch at Kronecker 2^22 against 756.)
__device__ __forceinline__ void long_row(const VerifyArgs &a, int64_t u, int lane) {
  const uint32_t lo = a.rowoff[u], hi = a.rowoff[u + 1];  // j + 63 may pass 2^31
  float sum = 0.f;
  float c = lo + lane < hi ? a.contrib[a.col[lo + lane]] : 0.f;
  for (uint32_t j = lo; j < hi; j += 32) {
    const int cnt = min(32u, hi - j);
    const uint32_t jn = j + 32 + lane;
    const float cn = jn < hi ? a.contrib[a.col[jn]] : 0.f;
    if (cnt == 32) {
#pragma unroll
      for (int k = 0; k < 32; k++) sum = __fadd_rn(sum, __shfl_sync(kFull, c, k));
    } else {
      for (int k = 0; k < cnt; k++) sum = __fadd_rn(sum, __shfl_sync(kFull, c, k));
    }
    c = cn;
  }
  if (lane == 0) residual(a, u, sum);
}

// A thread per row, the loads of four entries issued before their adds.
__device__ __forceinline__ void short_row(const VerifyArgs &a, int64_t u) {
  const int32_t lo = a.rowoff[u], hi = a.rowoff[u + 1];
  float sum = 0.f;
  int32_t j = lo;
  for (; j + 3 < hi; j += 4) {
    const float c0 = a.contrib[a.col[j]], c1 = a.contrib[a.col[j + 1]];
    const float c2 = a.contrib[a.col[j + 2]], c3 = a.contrib[a.col[j + 3]];
    sum = __fadd_rn(sum, c0);
    sum = __fadd_rn(sum, c1);
    sum = __fadd_rn(sum, c2);
    sum = __fadd_rn(sum, c3);
  }
  for (; j < hi; j++) sum = __fadd_rn(sum, a.contrib[a.col[j]]);
  residual(a, u, sum);
}

__global__ void __launch_bounds__(kVerifyThreads, 4) verify_rows_kernel(const VerifyArgs a) {
  __shared__ __align__(16) float buf[2][kHubChunk];
  if (blockIdx.x < a.nhub) {
    hub_row(a, buf);
    return;
  }
  const int64_t b = blockIdx.x - a.nhub;
  if (b < a.long_blocks) {
    const int64_t u = a.nhub + b * (kVerifyThreads / 32) + (threadIdx.x >> 5);
    if (u < a.nlong) long_row(a, u, threadIdx.x & 31);
    return;
  }
  const int64_t u = a.nlong + (b - a.long_blocks) * kVerifyThreads + threadIdx.x;
  if (u < a.n) short_row(a, u);
}

// ---- the residuals' sum -------------------------------------------------------
//
// The reference adds the residuals to a double one after the other; the
// rounding of each add depends on the sum before it, so the result is that of
// one order only.  It can be had in parallel all the same.  While the sum S
// stays within a binade [2^k, 2^(k+1)) its unit u = 2^(k-52) is fixed, S is a
// multiple of u and adding x >= 0 adds x / u rounded to an integer, whatever
// S is -- except when x / u lies halfway between two integers: then the even
// result is taken, which depends on the parity of S / u only.  So a run of
// residuals is a function of that parity, the pair of integers it adds for
// even and for odd S / u, and such functions compose associatively.  A plain
// prefix sum tells the binade of every run but those in which S passes a
// power of two (or might, within the prefix sum's error); these few are added
// one residual after the other.  The last kernel checks with the exact S that
// every run it takes as a whole begins and ends in its binade.

// What a run of residuals adds, in units of 2^(k - 52), for even / odd S.
struct Run {
  int k;  // binade; kNoRun: unknown, kZeroRun: adds nothing in any binade
  int64_t add[2];
};
constexpr int kNoRun = -100000, kZeroRun = 100000;

__device__ __forceinline__ Run join(const Run &x, const Run &y) {
  if (x.k == kZeroRun) return y;
  if (y.k == kZeroRun) return x;
  Run r;
  r.k = x.k == y.k ? x.k : kNoRun;
#pragma unroll
  for (int p = 0; p < 2; p++) r.add[p] = x.add[p] + y.add[(p + x.add[p]) & 1];
  return r;
}

// Adding x in binade k, q = x 2^(52 - k) (exact, a power of two).
__device__ __forceinline__ Run one(double q, int k) {
  const double fl = floor(q), rest = q - fl;
  // 2^53 units leave the binade; cut off so that sums of them stay in range
  const int64_t w = q < 9007199254740992.0 ? static_cast<int64_t>(fl) : int64_t(1) << 54;
  if (rest == 0.5) return Run{k, {w + (w & 1), w + ((w & 1) ^ 1)}};
  const int64_t r = w + (rest > 0.5);
  return Run{k, {r, r}};
}

// Exponent of a positive normal double, and 2^e (sums of floats, and what
// scales them, are normal).
__device__ __forceinline__ int binade(double x) {
  return ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
}
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double(static_cast<long long>(e + 1023) << 52);
}

// Plain sums of runs of kRunLen residuals, a warp each; *odd is set when a
// residual is infinite or NaN.
__global__ void __launch_bounds__(kVerifyThreads)
run_sums_kernel(int64_t n, int64_t nruns, const float *__restrict__ resid, double *sum, int *odd) {
  const int64_t r = (static_cast<int64_t>(blockIdx.x) * kVerifyThreads + threadIdx.x) >> 5;
  if (r >= nruns) return;
  const int lane = threadIdx.x & 31;
  double v = 0;
  for (int64_t i = r * kRunLen + lane; i < min(n, (r + 1) * kRunLen); i += 32) v += resid[i];
  v = warp_sum_d(v);
  if (lane == 0) {
    sum[r] = v;
    if (!isfinite(v)) atomicOr(odd, 1);
  }
}

// sum[r] = sum of the runs before r, sum[nruns] = all, by one block.
__global__ void __launch_bounds__(1024) run_prefix_kernel(int64_t nruns, double *sum) {
  __shared__ double part[1024];
  const int t = threadIdx.x;
  const int64_t per = (nruns + 1023) / 1024, lo = min(nruns, t * per), hi = min(nruns, lo + per);
  double v = 0;
  for (int64_t i = lo; i < hi; i++) v += sum[i];
  part[t] = v;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const double x = t >= o ? part[t - o] : 0.0;
    __syncthreads();
    part[t] += x;
    __syncthreads();
  }
  double before = t ? part[t - 1] : 0.0;
  for (int64_t i = lo; i < hi; i++) {
    const double x = sum[i];
    sum[i] = before;
    before += x;
  }
  if (t == 1023) sum[nruns] = part[1023];
}

// The runs as functions of parity, a warp each (a lane takes kRunLen / 32
// consecutive residuals), and of every 32 runs together, a block each.
__global__ void __launch_bounds__(1024)
run_build_kernel(int64_t n, int64_t nruns, const float *__restrict__ resid,
                 const double *__restrict__ before, Run *run, Run *group) {
  constexpr int kPer = kRunLen / 32;
  __shared__ Run s_run[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t r = static_cast<int64_t>(blockIdx.x) * 32 + wid;
  Run f{kZeroRun, {0, 0}};
  if (r < nruns) {
    const double lo = before[r], hi = before[r + 1];
    {
      // the prefix sum is within n 2^-53 < 2^-22 of the exact one
      const double slack = 1e-6;
      const int k = lo > 0 ? binade(lo * (1 - slack)) : kNoRun;
      const bool known = lo > 0 && binade(hi * (1 + slack)) == k;
      const double scale = known ? pow2(52 - k) : 1.0;
      Run mine{kZeroRun, {0, 0}};
#pragma unroll
      for (int i = 0; i < kPer; i++) {
        const int64_t j = r * kRunLen + lane * kPer + i;
        const double x = j < n ? static_cast<double>(resid[j]) : 0.0;
        if (x > 0) {
          mine = join(mine, known ? one(x * scale, k) : Run{kNoRun, {0, 0}});
        }
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {  // lane l: residuals of lanes l .. l + 2 o - 1
        Run y;
        y.k = __shfl_down_sync(kFull, mine.k, o);
        y.add[0] = __shfl_down_sync(kFull, mine.add[0], o);
        y.add[1] = __shfl_down_sync(kFull, mine.add[1], o);
        if ((lane & (2 * o - 1)) == 0) mine = join(mine, y);
      }
      f = mine;
    }
    if (lane == 0) run[r] = f;
  }
  if (lane == 0) s_run[wid] = f;
  __syncthreads();
  if (threadIdx.x == 0) {
    Run g = s_run[0];
    for (int i = 1; i < 32; i++) g = join(g, s_run[i]);
    group[blockIdx.x] = g;
  }
}

__device__ __forceinline__ Run shfl_up_run(const Run &x, int o) {
  return Run{__shfl_up_sync(kFull, x.k, o),
             {__shfl_up_sync(kFull, x.add[0], o), __shfl_up_sync(kFull, x.add[1], o)}};
}

// Takes the runs of lanes pos, pos + 1, ... up to the first that S does not
// begin and end in the binade of; returns its lane (32: none).  One warp.
__device__ __forceinline__ int take_runs(Run f, int pos, double &S, int lane) {
  const int k = S > 0 ? binade(S) : kNoRun;
  if (lane < pos) f = Run{kZeroRun, {0, 0}};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Run y = shfl_up_run(f, o);
    if (lane >= o) f = join(y, f);
  }
  int64_t e = 0;
  bool ok = f.k == kZeroRun;
  if (k != kNoRun) {
    e = static_cast<int64_t>(S * pow2(52 - k));
    if (!ok) {
      e += f.add[e & 1];
      ok = f.k == k && e < (int64_t(1) << 53);
    }
  }
  const unsigned out = __ballot_sync(kFull, lane >= pos && !ok);
  const int stop = out ? __ffs(out) - 1 : 32;
  const int64_t at = __shfl_sync(kFull, e, (stop + 31) & 31);
  if (stop > pos && k != kNoRun) S = static_cast<double>(at) * pow2(k - 52);
  return stop;
}

// S after kRunLen residuals among which it leaves its binade; one warp, a lane
// holding kPer consecutive ones.  The lanes' runs in S's present binade are
// taken up to the lane that leaves it, whose residuals are added one after
// the other; then again from the new binade.
template <int kPer>
__device__ __forceinline__ double slow_run(const float (&x)[kPer], double S, int lane) {
  int pos = 0;  // next lane
  while (pos < 32) {
    int stop = pos;
    if (S > 0) {
      const int k = binade(S);
      const double scale = pow2(52 - k);
      Run f{kZeroRun, {0, 0}};
#pragma unroll
      for (int i = 0; i < kPer; i++)
        if (x[i] > 0) f = join(f, one(static_cast<double>(x[i]) * scale, k));
      stop = take_runs(f, pos, S, lane);
    }
    if (stop < 32) {
      double t = S;
#pragma unroll
      for (int i = 0; i < kPer; i++) t += static_cast<double>(x[i]);
      S = __shfl_sync(kFull, t, stop);
    }
    pos = stop + 1;
  }
  return S;
}

// The exact sum, by one warp: groups of runs 32 at a time, the runs of a group
// that cannot be taken whole, and the residuals of such a run.
__global__ void __launch_bounds__(32)
run_total_kernel(int64_t n, int64_t nruns, const float *__restrict__ resid,
                 const double *__restrict__ before, const Run *__restrict__ run,
                 const Run *__restrict__ group, const int *__restrict__ odd, double *out) {
  constexpr int kPer = kRunLen / 32;
  const int lane = threadIdx.x;
  if (*odd) {  // an infinity or a NaN: any order gives the same
    if (lane == 0) *out = before[nruns];
    return;
  }
  const Run none{kZeroRun, {0, 0}};
  const int64_t ngroups = (nruns + 31) / 32;
  double S = 0;
  for (int64_t g0 = 0; g0 < ngroups; g0 += 32) {
    const Run f = g0 + lane < ngroups ? group[g0 + lane] : none;
    for (int g = 0; (g = take_runs(f, g, S, lane)) < 32; g++) {
      const int64_t r0 = (g0 + g) * 32;
      const Run h = r0 + lane < nruns ? run[r0 + lane] : none;
      for (int r = 0; (r = take_runs(h, r, S, lane)) < 32; r++) {
        const int64_t j = (r0 + r) * kRunLen + lane * kPer;
        float x[kPer];
#pragma unroll
        for (int i = 0; i < kPer; i++) x[i] = j + i < n ? resid[j + i] : 0.f;
        S = slow_run(x, S, lane);
      }
    }
  }
  if (lane == 0) *out = S;
}

}  // namespace

cudaError_t VerifyResiduals(const DeviceGraph &g, const float *score_orig, float damping,
                            float *contrib, float *resid_orig, cudaStream_t s) {
  const int64_t n = g.n;
  if (n < 1) return cudaSuccess;
  // the reference's base score: (1 - d) / N in float, N converted to float
  const float base = (1.0f - damping) / static_cast<float>(n);
  verify_contrib_kernel<<<static_cast<unsigned>((n + kVerifyThreads - 1) / kVerifyThreads),
                          kVerifyThreads, 0, s>>>(n, score_orig, g.perm, g.rowoff,
                                                  g.directed ? g.odeg : nullptr, contrib);
  // hub and long rows: the degree bins of at least 4,096 and of at
  // least kLongRow entries (the split only decides who adds a row, never the result)
  int b = 0;
  while (b < kBinZero && g.bins.min_len[b] >= kLongRow) b++;
  VerifyArgs a;
  a.n = n;
  a.nhub = g.bin_row_start[1];
  a.nlong = std::min<int64_t>(n, g.bin_row_start[b]);
  a.long_blocks = static_cast<unsigned>((a.nlong - a.nhub + kVerifyThreads / 32 - 1) /
                                        (kVerifyThreads / 32));
  a.rowoff = g.rowoff;
  a.col = g.col;
  a.contrib = contrib;
  a.score_orig = score_orig;
  a.perm = g.perm;
  a.base = base;
  a.damping = damping;
  a.resid_orig = resid_orig;
  const int64_t blocks = a.nhub + a.long_blocks + (n - a.nlong + kVerifyThreads - 1) / kVerifyThreads;
  verify_rows_kernel<<<static_cast<unsigned>(blocks), kVerifyThreads, 0, s>>>(a);
  return cudaGetLastError();
}

void FreeVerifyScratch(VerifyScratch *v) {
  if (v->mem) cudaFree(v->mem);
  *v = VerifyScratch();
}

cudaError_t SumInOrder(int64_t n, const float *resid, VerifyScratch &v, double *out,
                       cudaStream_t s) {
  const int64_t nruns = (n + kRunLen - 1) / kRunLen, ngroups = (nruns + 31) / 32;
  // out, odd, before, run, group
  const size_t off_before = 16;
  const size_t off_run = off_before + sizeof(double) * ((nruns + 2) & ~int64_t(1));
  const size_t bytes = off_run + sizeof(Run) * (nruns + ngroups);
  cudaError_t e = cudaSuccess;
  if (v.bytes < bytes) {
    FreeVerifyScratch(&v);
    e = cudaMalloc(&v.mem, bytes);
    if (e != cudaSuccess) return e;
    v.bytes = bytes;
  }
  char *p = static_cast<char *>(v.mem);
  double *total = reinterpret_cast<double *>(p);
  int *odd = reinterpret_cast<int *>(p + 8);
  double *before = reinterpret_cast<double *>(p + off_before);
  Run *run = reinterpret_cast<Run *>(p + off_run), *group = run + nruns;
  e = cudaMemsetAsync(p, 0, 16, s);
  if (e != cudaSuccess) return e;
  const unsigned wb = static_cast<unsigned>((nruns + kVerifyThreads / 32 - 1) / (kVerifyThreads / 32));
  run_sums_kernel<<<wb, kVerifyThreads, 0, s>>>(n, nruns, resid, before, odd);
  run_prefix_kernel<<<1, 1024, 0, s>>>(nruns, before);
  run_build_kernel<<<static_cast<unsigned>(ngroups), 1024, 0, s>>>(n, nruns, resid, before, run, group);
  run_total_kernel<<<1, 32, 0, s>>>(n, nruns, resid, before, run, group, odd, total);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, total, sizeof(double), cudaMemcpyDeviceToHost, s);
  return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}

}  // namespace prgpu
