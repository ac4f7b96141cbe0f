// bfs.cu -- direction-optimizing breadth-first search on the device CSR
// mirror (pr_gpu_bfs in include/pr_gpu.h).
//
// The reference's DOBFS (src/bfs.cc:38-174), step for step:
//   * the source is its own parent;
//   * top-down step: every frontier vertex claims its unvisited
//     out-neighbours by compare-and-swap on parent[], the claimed vertices
//     form the next frontier queue, and the step returns the scout count
//     (the summed out-degrees of the claimed vertices, 1 for a vertex
//     without out-edges: the reference starts parent[v] at -out_degree(v),
//     or -1, and adds the negated parent it replaced; here unvisited parents
//     are all -1, set by one memset, and the degree is read at the claim);
//   * bottom-up step: every unvisited vertex takes the first in-neighbour
//     found in the frontier bitmap as its parent, the found vertices form the
//     next bitmap, and the step returns their number;
//   * the same switching rule: top-down while scout_count <= edges_to_check /
//     alpha (edges_to_check starts at M and loses each top-down step's scout
//     count), bottom-up while the awake count grows or stays above N / beta,
//     then back to a queue (alpha = 15, beta = 18);
//   * unvisited vertices end with parent -1.
// One cooperative launch does a whole search: init, the steps, the write-back,
// with a grid barrier (grid_barrier.cuh) between the phases.  After each step
// every CTA applies the switching rule to the same counts, so all choose the
// same next step.  (As kernels of a conditional graph the steps cost about
// 10 us each beside their work: 428 us a search of Kronecker 2^23 in 9 steps,
// 177 us on 1,000 vertices; 269 and 68 in one launch.)  1024-thread CTAs,
// two per SM: 32 registers a thread, as many warps as an SM holds, since the
// bottom-up step is bound by its chains of dependent loads.
// Queues and bitmaps hold the mirror's degree-sorted ids; parent[] is
// indexed by mirror row but stores the parent's original id, so the
// write-back only gathers it into original order.
// Parents can differ from run to run (which frontier vertex wins a claim is
// a race, as in the reference); depths, reached sets and tree sizes cannot.
//
// Top-down work is spread over the frontier's edges, not its vertices
// (frontier degrees are scanned, each thread takes edges and finds its
// vertex by a forward search in the scan), so a hub in the frontier does not
// serialise a warp.  Bottom-up work: each warp owns two words of 32
// consecutive vertices at a time, walks the two vertices of every lane
// together, and writes each bitmap word with one ballot.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "grid_barrier.cuh"
#include "internal.h"

namespace prgpu {

namespace {

// Step kinds.
enum BfsKind : int32_t {
  kTdSmall,   // "td", frontier scanned inside each block
  kTdBig,     // "td", frontier scanned device-wide
  kToBitmap,  // "e": queue -> bitmap (entering bottom-up)
  kBottomUp,  // "bu"
  kToQueue,   // "c": bitmap -> queue (leaving bottom-up)
  kDone,      // the search ends
  kInit,      // "i": the source set-up
};

constexpr int kThreads = 1024, kWarps = kThreads / 32, kCtasPerSm = 2;
constexpr unsigned kFull = 0xffffffffu;

constexpr int kBfsMaxLog = 1024;  // logged steps (the count goes on beyond)

struct BfsCounters {
  unsigned long long qtail;  // next-frontier queue length
  unsigned long long scout;  // top-down scout count
  unsigned long long awake;  // bottom-up awake count
};

struct BfsLogRec {
  int32_t kind;
  int32_t unused;
  int64_t count;
  unsigned long long ns;
};

// In device memory.  Step i adds to cnt[i % 3]; cnt[(i + 1) % 3] is cleared
// during it, a slot all CTAs read two steps before.
struct BfsCtl {
  GridBarrier barrier;
  BfsCounters cnt[3];
  BfsLogRec log[kBfsMaxLog];
};

// Search state; every CTA keeps the same one.
struct BfsState {
  int32_t next;   // the step to run
  int32_t mode;   // 0: frontier in a queue (top-down), 1: in a bitmap
  int32_t cur;    // queue[cur] is the frontier
  int32_t front;  // bm[front] is the frontier bitmap
  int32_t used;   // bitmaps written since they were cleared
  int32_t nlog;   // steps logged (all steps, also past kBfsMaxLog)
  int64_t qsize, edges_to_check, scout, awake, old_awake, guard;
  unsigned long long t_prev;
};

struct BfsArgs {
  BfsCtl *ctl;
  BfsResult *res;
  int32_t *q0, *q1, *parent;
  unsigned *bm0, *bm1;
  int32_t *eoff, *sums;
  const int32_t *__restrict__ ooff;
  const int32_t *__restrict__ onbr;
  const int32_t *__restrict__ ioff;
  const int32_t *__restrict__ inbr;
  const int32_t *__restrict__ perm;
  const int32_t *__restrict__ inv;
  int32_t *out_old;
  int64_t m;
  int32_t n, in_rows, hub_rows, source_old, alpha, beta;
  unsigned max_polls;
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int32_t out_degree(const int32_t *ooff, int v) {
  return ooff[v + 1] - ooff[v];
}

// Folds the step that just ran into the state (src/bfs.cc:140-172), logs it,
// and picks the next one by the reference's rule; the step guard ends the
// search after at most n + 2 steps whatever the counts say.  Thread 0.
__device__ __forceinline__ void decide(const BfsArgs &a, BfsState &c, int step) {
  const BfsCounters *cnt = &a.ctl->cnt[(step + 2) % 3];  // of the step before
  const int64_t n = a.n;
  const int last = c.next;
  int64_t count = -1;
  switch (last) {
    case kTdSmall:
    case kTdBig:
      c.scout = static_cast<int64_t>(__ldcg(&cnt->scout));
      c.qsize = static_cast<int64_t>(__ldcg(&cnt->qtail));
      c.cur ^= 1;
      count = c.qsize;
      break;
    case kToBitmap:
      c.awake = c.qsize;
      c.front = 0;
      c.used = 1;
      break;
    case kBottomUp:
      c.awake = static_cast<int64_t>(__ldcg(&cnt->awake));
      c.front ^= 1;
      count = c.awake;
      break;
    case kToQueue:
      c.qsize = static_cast<int64_t>(__ldcg(&cnt->qtail));
      c.scout = 1;
      c.mode = 0;
      break;
    default:  // kInit
      break;
  }
  if (blockIdx.x == 0) {
    const unsigned long long now = global_ns();
    if (c.nlog < kBfsMaxLog) a.ctl->log[c.nlog] = BfsLogRec{last, 0, count, now - c.t_prev};
    c.t_prev = now;
  }
  c.nlog++;
  int next;
  if (c.mode == 1) {
    if (last == kToBitmap || c.awake >= c.old_awake || c.awake > n / a.beta) {
      c.old_awake = c.awake;
      next = kBottomUp;
    } else {
      next = kToQueue;
    }
  } else if (c.qsize == 0) {
    next = kDone;
  } else if (c.scout > c.edges_to_check / a.alpha) {
    c.mode = 1;
    next = kToBitmap;
  } else {
    c.edges_to_check -= c.scout;
    next = c.qsize <= kThreads ? kTdSmall : kTdBig;
  }
  if (next != kDone && ++c.guard > n + 2) {
    if (blockIdx.x == 0) a.res->error = 1;
    next = kDone;
  }
  c.next = next;
}

// Exclusive block-wide scan of one value per thread; *total: the sum.  Called
// by all threads; s_warp: kWarps words.
template <typename T>
__device__ __forceinline__ T block_scan(T v, T *s_warp, T *total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();  // s_warp may still be read
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  T w = s_warp[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(kFull, w, o);
    if (lane >= o) w += t;
  }
  *total = __shfl_sync(kFull, w, 31);
  const T before = __shfl_sync(kFull, w, (wid + 31) & 31);
  return (wid ? before : T(0)) + incl - v;
}

// Where this thread's `mine` values go in the queue: one global atomic per
// block reserves the block's run.  Called by all threads.
__device__ __forceinline__ unsigned long long reserve(int mine, unsigned long long *tail,
                                                      int *s_warp, unsigned long long *s_base) {
  int total;
  const int pre = block_scan(mine, s_warp, &total);
  if (threadIdx.x == 0)
    *s_base = total ? atomicAdd(tail, static_cast<unsigned long long>(total)) : 0ull;
  __syncthreads();
  return *s_base + pre;
}

// ---- top-down ----------------------------------------------------------------

constexpr int kScanChunk = 2 * kThreads;
constexpr int64_t kEntriesPerCta = 4096;
constexpr int kMaxPerThread = 8;

// Exclusive scan of the frontier's out-degrees, chunk by chunk: eoff[i] within
// the chunk, the chunk's total to sums[].
__device__ __forceinline__ void scan_chunks(const BfsArgs &a, const BfsState &c, int *s_warp) {
  const int32_t *queue = c.cur ? a.q1 : a.q0;
  const int64_t items = c.qsize + 1;  // one past the last: the edge count
  const int64_t nch = (items + kScanChunk - 1) / kScanChunk;
  for (int64_t k = blockIdx.x; k < nch; k += gridDim.x) {
    const int64_t i = k * kScanChunk + 2 * threadIdx.x;
    const int d0 = i < c.qsize ? out_degree(a.ooff, queue[i]) : 0;
    const int d1 = i + 1 < c.qsize ? out_degree(a.ooff, queue[i + 1]) : 0;
    int total;
    const int pre = block_scan(d0 + d1, s_warp, &total);
    if (i < items) a.eoff[i] = pre;
    if (i + 1 < items) a.eoff[i + 1] = pre + d0;
    if (threadIdx.x == 0) a.sums[k] = total;
  }
}

// The chunks' totals become what comes before them; one block.
__device__ __forceinline__ void scan_sums(const BfsArgs &a, const BfsState &c, int *s_warp) {
  const int64_t nch = (c.qsize + 1 + kScanChunk - 1) / kScanChunk;
  const int64_t per = (nch + kThreads - 1) / kThreads;
  const int64_t lo = min(nch, per * threadIdx.x), hi = min(nch, lo + per);
  int run = 0;
  for (int64_t i = lo; i < hi; i++) run += a.sums[i];
  int total;
  int pre = block_scan(run, s_warp, &total);
  for (int64_t i = lo; i < hi; i++) {
    const int x = a.sums[i];
    a.sums[i] = pre;
    pre += x;
  }
}

// Top-down step over the frontier's edges: edge e belongs to the frontier
// vertex i with off(i) <= e < off(i + 1) (off: exclusive scan of the
// frontier's out-degrees, off(q) = edges).  Each block takes chunks of
// kThreads * per consecutive edges; a thread's edges are kThreads apart, so
// its frontier index only moves forward and is re-searched only when it
// passes the current vertex.  SMALL (q <= kThreads): every block scans the
// frontier's degrees itself in shared memory, so a small step is one phase.
template <bool SMALL>
__device__ __forceinline__ void top_down(const BfsArgs &a, const BfsState &c, BfsCounters *cnt,
                                         int32_t *s_eoff, int32_t *s_q, int *s_warp,
                                         unsigned long long *s_base) {
  const int32_t *queue = c.cur ? a.q1 : a.q0;
  int32_t *next = c.cur ? a.q0 : a.q1;
  const int q = static_cast<int>(c.qsize);
  if (SMALL) {
    int u = 0, d = 0;
    if (threadIdx.x < q) {
      u = queue[threadIdx.x];
      d = out_degree(a.ooff, u);
    }
    int total;
    const int pre = block_scan(d, s_warp, &total);
    s_eoff[threadIdx.x] = pre;
    s_q[threadIdx.x] = u;
    if (threadIdx.x == 0) s_eoff[kThreads] = total;
    __syncthreads();
  }
  auto off = [&](int i) { return SMALL ? s_eoff[i] : a.eoff[i] + a.sums[i / kScanChunk]; };
  const int64_t edges = SMALL ? s_eoff[kThreads] : off(q);
  // small steps: fewer edges a thread, so that every block has some
  const int64_t wave = static_cast<int64_t>(gridDim.x) * kThreads;
  const int per = static_cast<int>(min(static_cast<int64_t>(kMaxPerThread), (edges + wave - 1) / wave));
  unsigned long long scout = 0;
  int lo = 0;  // frontier index of this thread's previous edge
  int end = 0, begin = 0;  // its edges
  if (edges > 0) {
    begin = off(0);
    end = off(1);
  }
  for (int64_t c0 = static_cast<int64_t>(blockIdx.x) * kThreads * per; c0 < edges;
       c0 += wave * per) {
    int vals[kMaxPerThread];
    unsigned mask = 0;
#pragma unroll
    for (int k = 0; k < kMaxPerThread; k++) {
      const int64_t e = c0 + k * kThreads + threadIdx.x;
      vals[k] = 0;
      if (k < per && e < edges) {
        if (end <= e) {  // past vertex lo: last i with off(i) <= e
          int l = lo + 1, h = q - 1;
          while (l < h) {
            const int mid = (l + h + 1) >> 1;
            if (off(mid) <= e) l = mid;
            else h = mid - 1;
          }
          lo = l;
          begin = off(lo);
          end = off(lo + 1);
        }
        const int u = SMALL ? s_q[lo] : queue[lo];
        const int v = a.onbr[a.ooff[u] + (static_cast<int>(e) - begin)];
        // a weak load that L1 may serve (the popular targets are hubs read
        // by every block): a parent never returns to -1, so a value >= 0 is
        // final, and a stale -1 only costs a compare-and-swap that fails
        int32_t curp;
        asm volatile("ld.global.ca.s32 %0, [%1];" : "=r"(curp) : "l"(a.parent + v));
        if (curp < 0 && atomicCAS(a.parent + v, -1, __ldg(a.perm + u)) == -1) {
          vals[k] = v;
          mask |= 1u << k;
          scout += static_cast<unsigned long long>(max(out_degree(a.ooff, v), 1));
        }
      }
    }
    unsigned long long pos = reserve(__popc(mask), &cnt->qtail, s_warp, s_base);
#pragma unroll
    for (int k = 0; k < kMaxPerThread; k++)
      if ((mask >> k) & 1u) next[pos++] = vals[k];
  }
  for (int o = 16; o > 0; o >>= 1) scout += __shfl_xor_sync(kFull, scout, o);
  if ((threadIdx.x & 31) == 0 && scout) atomicAdd(&cnt->scout, scout);
}

// ---- bottom-up -----------------------------------------------------------------

__device__ __forceinline__ bool in_front(const unsigned *front, int u) {
  return (front[u >> 5] >> (u & 31)) & 1u;
}

// The bottom-up step of this warp's words with hub rows (at least 4,096
// in-neighbours) in them.  A lane alone takes a microsecond an entry while all
// other CTAs wait at the barrier, so it walks the first kLaneWalk entries of
// its list (nearly all rows are found there) and the whole warp, 128 entries
// at a time, the rest of the lists left, one after the other.  Returns how
// many were found.  Apart from the loop over the other words it costs 0.4 % of
// a search of Kronecker 2^23 (228.7 us without, 229.6), inside it 2 to 9 %.
constexpr int kLaneWalk = 512;
__device__ __forceinline__ unsigned bottom_up_hubs(const BfsArgs &a, const unsigned *front,
                                                   unsigned *next, int warp, int warps) {
  const int lane = threadIdx.x & 31;
  unsigned awake = 0;
  for (int w = warp; w << 5 < a.hub_rows; w += warps) {
    const int v = (w << 5) + lane;
    int p = -1;  // the in-neighbour found (mirror row), if any
    bool left = v < a.in_rows && a.parent[v] < 0;
    if (left) {
      int j = a.ioff[v];
      const int len = a.ioff[v + 1] - j, e = j + min(len, kLaneWalk);
      for (; j < e && p < 0; j++) {
        const int u = a.inbr[j];
        if (in_front(front, u)) p = u;
      }
      left = p < 0 && len > kLaneWalk;
    }
    unsigned todo = __ballot_sync(kFull, left);
    while (todo) {
      const int b = __ffs(todo) - 1;
      todo &= todo - 1;
      const int row = (w << 5) + b;
      const unsigned end = a.ioff[row + 1];  // j + 128 may pass 2^31
      int found = -1;
      for (unsigned j = a.ioff[row] + kLaneWalk; j < end && found < 0; j += 128) {
        int u[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          u[k] = j + 32 * k + lane < end ? a.inbr[j + 32 * k + lane] : -1;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const unsigned hit = __ballot_sync(kFull, u[k] >= 0 && in_front(front, u[k]));
          if (hit && found < 0) found = __shfl_sync(kFull, u[k], __ffs(hit) - 1);
        }
      }
      if (lane == b) p = found;
    }
    if (p >= 0) a.parent[v] = __ldg(a.perm + p);
    const unsigned word = __ballot_sync(kFull, p >= 0);
    if (lane == 0) next[w] = word;
    awake += __popc(word);
  }
  return awake;
}

// Bottom-up step: each warp owns two bitmap words (32 consecutive vertices
// each) at a time and every lane walks its two vertices' in-lists together,
// so two independent load chains (neighbour id, then its frontier bit) are
// in flight per lane; each vertex still takes the first in-neighbour in list
// order found in the frontier.  Only rows [0, in_rows) have in-neighbours
// (rows are sorted by in-degree), so only their words are visited; the words
// after them stay zero.
__device__ __forceinline__ void bottom_up(const BfsArgs &a, const BfsState &c, BfsCounters *cnt) {
  const unsigned *front = c.front ? a.bm1 : a.bm0;
  unsigned *next = c.front ? a.bm0 : a.bm1;
  const int n = a.in_rows;
  const int lane = threadIdx.x & 31;
  const int words = static_cast<int>((static_cast<int64_t>(n) + 31) >> 5);
  const int warps = gridDim.x * kWarps;
  unsigned awake = 0;
  int w = blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (w << 5 < a.hub_rows) {
    awake = bottom_up_hubs(a, front, next, w, warps);
    while (w << 5 < a.hub_rows) w += warps;
  }
  for (; w < words; w += 2 * warps) {
    const int w2 = w + warps;  // the warp's second word (warp-uniform test)
    const int v1 = (w << 5) + lane, v2 = (w2 << 5) + lane;
    int j1 = 0, e1 = 0, j2 = 0, e2 = 0;
    if (v1 < n && a.parent[v1] < 0) {
      j1 = a.ioff[v1];
      e1 = a.ioff[v1 + 1];
    }
    if (w2 < words && v2 < n && a.parent[v2] < 0) {
      j2 = a.ioff[v2];
      e2 = a.ioff[v2 + 1];
    }
    int p1 = -1, p2 = -1;  // the in-neighbour found (mirror row), if any
    while (j1 < e1 || j2 < e2) {
      const int u1 = j1 < e1 ? a.inbr[j1] : -1;
      const int u2 = j2 < e2 ? a.inbr[j2] : -1;
      const bool h1 = u1 >= 0 && in_front(front, u1);
      const bool h2 = u2 >= 0 && in_front(front, u2);
      if (h1) {
        p1 = u1;
        e1 = j1;  // chain 1 done
      } else {
        j1++;
      }
      if (h2) {
        p2 = u2;
        e2 = j2;
      } else {
        j2++;
      }
    }
    if (p1 >= 0) a.parent[v1] = __ldg(a.perm + p1);
    if (p2 >= 0) a.parent[v2] = __ldg(a.perm + p2);
    const unsigned word1 = __ballot_sync(kFull, p1 >= 0);
    if (lane == 0) next[w] = word1;
    awake += __popc(word1);
    if (w2 < words) {
      const unsigned word2 = __ballot_sync(kFull, p2 >= 0);
      if (lane == 0) next[w2] = word2;
      awake += __popc(word2);
    }
  }
  if (lane == 0 && awake) atomicAdd(&cnt->awake, static_cast<unsigned long long>(awake));
}

// Set bits of the frontier bitmap -> queue[cur], over the words of the rows
// with in-edges, one word per thread and block round.
__device__ __forceinline__ void bitmap_to_queue(const BfsArgs &a, const BfsState &c,
                                                BfsCounters *cnt, int *s_warp,
                                                unsigned long long *s_base) {
  const unsigned *bm = c.front ? a.bm1 : a.bm0;
  int32_t *queue = c.cur ? a.q1 : a.q0;
  const int64_t words = (static_cast<int64_t>(a.in_rows) + 31) >> 5;
  for (int64_t w0 = static_cast<int64_t>(blockIdx.x) * kThreads; w0 < words;
       w0 += static_cast<int64_t>(gridDim.x) * kThreads) {
    const int64_t w = w0 + threadIdx.x;
    unsigned word = 0;
    if (w < words) {
      word = bm[w];
      const int64_t rest = static_cast<int64_t>(a.in_rows) - (w << 5);
      if (rest < 32) word &= (1u << rest) - 1u;
    }
    unsigned long long pos = reserve(__popc(word), &cnt->qtail, s_warp, s_base);
    while (word) {
      const int b = __ffs(word) - 1;
      word &= word - 1u;
      queue[pos++] = static_cast<int32_t>((w << 5) + b);
    }
  }
}

__device__ __forceinline__ void clear_bitmaps(const BfsArgs &a, int64_t gtid, int64_t gthreads) {
  const int64_t words = (static_cast<int64_t>(a.n) + 31) >> 5;
  for (int64_t i = gtid; i < words; i += gthreads) a.bm0[i] = a.bm1[i] = 0u;
}

__global__ void __launch_bounds__(kThreads, kCtasPerSm) bfs_kernel(const BfsArgs a) {
  __shared__ int32_t s_eoff[kThreads + 1], s_q[kThreads];
  __shared__ int s_warp[32];
  __shared__ unsigned long long s_base;
  __shared__ BfsState st;
  __shared__ int s_ok;
  const int64_t gthreads = static_cast<int64_t>(gridDim.x) * kThreads;
  const int64_t gtid = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  unsigned round = 0;
  auto barrier = [&] {
    const bool ok = grid_barrier(&a.ctl->barrier, ++round, a.max_polls, &s_ok);
    if (!ok && threadIdx.x == 0) a.res->error = 2;
    return ok;
  };

  // the source (original id) becomes its own parent and the first frontier;
  // its out-degree is the first scout count.  parent[] is indexed by mirror
  // row but holds original ids (only its sign is read during the search), so
  // the write-back needs no second lookup.
  const int src = a.inv[a.source_old];
  for (int64_t i = gtid; i < a.n; i += gthreads) a.parent[i] = i == src ? a.source_old : -1;
  clear_bitmaps(a, gtid, gthreads);
  if (gtid == 0) {
    a.q0[0] = src;
    a.ctl->cnt[0] = BfsCounters{0, 0, 0};
  }
  if (threadIdx.x == 0) {
    st = BfsState{kInit, 0, 0, 0, 0, 0, 1, a.m, out_degree(a.ooff, src), 0, 0, 0, 0};
    if (blockIdx.x == 0) st.t_prev = global_ns();
  }
  if (!barrier()) return;

  for (int step = 0;; step++) {
    if (threadIdx.x == 0) decide(a, st, step);
    __syncthreads();
    const int kind = st.next;
    if (kind == kDone) break;
    BfsCounters *cnt = &a.ctl->cnt[step % 3];
    if (gtid == 0) a.ctl->cnt[(step + 1) % 3] = BfsCounters{0, 0, 0};
    if (kind == kTdSmall) {
      top_down<true>(a, st, cnt, s_eoff, s_q, s_warp, &s_base);
    } else if (kind == kTdBig) {
      scan_chunks(a, st, s_warp);
      if (!barrier()) return;
      if (blockIdx.x == 0) scan_sums(a, st, s_warp);
      if (!barrier()) return;
      top_down<false>(a, st, cnt, s_eoff, s_q, s_warp, &s_base);
    } else if (kind == kToBitmap) {
      if (st.used) {  // bottom-up a second time
        clear_bitmaps(a, gtid, gthreads);
        if (!barrier()) return;
      }
      const int32_t *queue = st.cur ? a.q1 : a.q0;
      for (int64_t i = gtid; i < st.qsize; i += gthreads) {
        const int v = queue[i];
        atomicOr(a.bm0 + (v >> 5), 1u << (v & 31));
      }
    } else if (kind == kBottomUp) {
      // a source without in-edges has the only bit past the rows that
      // bottom-up steps write; it is spent once bm0 has been read
      if (gtid == 0 && st.front == 1 && (src >> 5) >= ((a.in_rows + 31) >> 5)) a.bm0[src >> 5] = 0u;
      bottom_up(a, st, cnt);
    } else {
      bitmap_to_queue(a, st, cnt, s_warp, &s_base);
    }
    if (!barrier()) return;
  }

  // Parents in original ids, -1 for unreached: each original id gathers its
  // row's parent (coalesced writes).  Rows [in_rows, n) have no in-edges, so
  // only the source among them is reached; their parents are not read.
  for (int64_t o = gtid; o < a.n; o += gthreads) {
    const int v = a.inv[o];
    int32_t r = -1;
    if (v < a.in_rows) r = a.parent[v];
    else if (o == a.source_old) r = a.source_old;
    a.out_old[o] = r;
  }
  if (gtid == 0) a.res->nlog = st.nlog;
  leave_grid(&a.ctl->barrier);
}

const char *StepName(int kind) {
  switch (kind) {
    case kInit: return "i";
    case kTdSmall:
    case kTdBig: return "td";
    case kToBitmap: return "e";
    case kBottomUp: return "bu";
    case kToQueue: return "c";
    default: return "?";
  }
}

}  // namespace

void FreeBfsScratch(BfsScratch *b) {
  void *ptrs[] = {b->parent, b->queue[0], b->queue[1], b->bm[0], b->bm[1], b->eoff, b->sums,
                  b->ctl};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (b->res) cudaFreeHost(b->res);
  *b = BfsScratch();
}

#define BFS_TRY(expr)                                                  \
  do {                                                                 \
    cudaError_t e_ = (expr);                                           \
    if (e_ != cudaSuccess) {                                           \
      *err = std::string("bfs: ") + #expr + ": " + cudaGetErrorString(e_); \
      return e_;                                                       \
    }                                                                  \
  } while (0)

cudaError_t BreadthFirstSearch(const DeviceGraph &g, BfsScratch &b, cudaStream_t s,
                               int source_old, int alpha, int beta, unsigned max_polls,
                               int32_t *out_old,
                               std::vector<BfsStep> *steps, int64_t *nsteps,
                               std::string *err) {
  const int64_t n = g.n;
  const int64_t words = (n + 31) / 32;
  const int64_t nch = (n + 1 + kScanChunk - 1) / kScanChunk;
  if (!b.parent || b.cap_n < n) {
    FreeBfsScratch(&b);
    BFS_TRY(cudaMalloc(&b.parent, sizeof(int32_t) * std::max<int64_t>(n, 1)));
    BFS_TRY(cudaMalloc(&b.queue[0], sizeof(int32_t) * std::max<int64_t>(n, 1)));
    BFS_TRY(cudaMalloc(&b.queue[1], sizeof(int32_t) * std::max<int64_t>(n, 1)));
    BFS_TRY(cudaMalloc(&b.eoff, sizeof(int32_t) * (n + 1)));
    BFS_TRY(cudaMalloc(&b.sums, sizeof(int32_t) * (nch + 1)));
    BFS_TRY(cudaMalloc(&b.bm[0], sizeof(unsigned) * std::max<int64_t>(words, 1)));
    BFS_TRY(cudaMalloc(&b.bm[1], sizeof(unsigned) * std::max<int64_t>(words, 1)));
    BFS_TRY(cudaMalloc(&b.ctl, sizeof(BfsCtl)));
    BFS_TRY(cudaMemsetAsync(b.ctl, 0, sizeof(BfsCtl), s));
    BFS_TRY(cudaHostAlloc(reinterpret_cast<void **>(&b.res), sizeof(BfsResult),
                          cudaHostAllocMapped | cudaHostAllocPortable));
    b.cap_n = n;
  }
  BfsArgs a;
  std::memset(&a, 0, sizeof(a));
  a.ctl = static_cast<BfsCtl *>(b.ctl);
  a.res = b.res;
  a.q0 = b.queue[0];
  a.q1 = b.queue[1];
  a.parent = b.parent;
  a.bm0 = b.bm[0];
  a.bm1 = b.bm[1];
  a.eoff = b.eoff;
  a.sums = b.sums;
  a.ooff = g.directed ? g.orowoff : g.rowoff;
  a.onbr = g.directed ? g.ocol : g.col;
  a.ioff = g.rowoff;
  a.inbr = g.col;
  a.perm = g.perm;
  a.inv = g.inv;
  a.out_old = out_old;
  a.m = g.m;
  a.n = static_cast<int32_t>(n);
  // in-CSR rows with in-neighbours (rows are sorted by in-degree; the rest
  // can only be reached as the source)
  a.in_rows = static_cast<int32_t>(g.bin_row_start[kBinZero]);
  a.hub_rows = static_cast<int32_t>(std::min(g.bin_row_start[1], g.bin_row_start[kBinZero]));
  a.source_old = source_old;
  a.max_polls = max_polls;
  a.alpha = alpha;
  a.beta = beta;
  int dev = 0, sms = 148;
  BFS_TRY(cudaGetDevice(&dev));
  BFS_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // a barrier is cheaper between fewer CTAs: one per kEntriesPerCta entries
  const int64_t want = std::max<int64_t>(1, (g.m + n) / kEntriesPerCta);
  const int grid = static_cast<int>(std::min<int64_t>(int64_t(sms) * kCtasPerSm, want));
  std::memset(b.res, 0, sizeof(BfsResult));
  BFS_TRY(LaunchGrid(reinterpret_cast<const void *>(bfs_kernel), grid, kThreads, &a, 0, s));
  BFS_TRY(cudaStreamSynchronize(s));
  const BfsResult *head = b.res;
  if (head->error) {
    const bool step_limit = head->error == 1;
    cudaMemsetAsync(b.ctl, 0, sizeof(BfsCtl), s);
    *err = step_limit ? "bfs: step limit exceeded" : "bfs: a grid barrier ran out of its wait";
    return cudaErrorUnknown;
  }
  if (nsteps) *nsteps = head->nlog;
  if (steps) {
    const int k = std::min<int>(head->nlog, kBfsMaxLog);
    std::vector<BfsLogRec> log(k);
    if (k > 0) {
      BFS_TRY(cudaMemcpyAsync(log.data(), a.ctl->log, sizeof(BfsLogRec) * k,
                              cudaMemcpyDeviceToHost, s));
      BFS_TRY(cudaStreamSynchronize(s));
    }
    steps->clear();
    for (const BfsLogRec &r : log)
      steps->push_back(BfsStep{StepName(r.kind), r.count, static_cast<double>(r.ns) * 1e-9});
  }
  return cudaSuccess;
}

#undef BFS_TRY

}  // namespace prgpu
