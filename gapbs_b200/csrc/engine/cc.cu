// cc.cu -- connected components on the device CSR mirror
// (pr_gpu_connected_components in include/pr_gpu.h).
//
// The reference's Afforest (src/cc.cc:40-150) labels every vertex with the
// root of its component tree; its Link always hooks the larger root under
// the smaller one and Compress only shortens chains, so every label is at
// most the vertex's own id and the final root of a component is its
// smallest vertex id.  That labelling is canonical, and the device computes
// exactly it:
//   1. comp[v] = v;
//   2. two sampling rounds: every vertex links with its r-th out-neighbour
//      (r = 0, 1), each round followed by a compress (which keeps the next
//      round's link chases short);
//   3. the component of the highest-degree vertex (row 0 of the degree-sorted
//      mirror: a vertex of the largest intermediate component, which the
//      reference estimates by sampling) is skipped in the final phase; row 0
//      has the smallest id, so it is the root of its tree and that
//      component's label is 0;
//   4. every other vertex links with its remaining out-neighbours and, for a
//      directed graph, with all its in-neighbours; compress;
//   5. ids are mapped back: each root takes the smallest original id of its
//      component (atomicMin; the largest component's members reduced per
//      block first), every vertex that root's label; a vertex without edges
//      is its own component and keeps its own id.
// Link is the reference's lock-free hooking loop with compare-and-swap; it
// and the compress chase are bounded (an iteration limit sets an error flag
// instead of spinning), so a defect cannot hang the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <string>

#include "grid_barrier.cuh"
#include "internal.h"

namespace prgpu {

namespace {

constexpr int kThreads = 1024, kCtasPerSm = 2;
constexpr unsigned kLongList = 32;  // entries of a row that a warp links together
constexpr int kChaseLimit = 1 << 20;  // far above any tree depth reached

__device__ __forceinline__ int ld_comp(const int *comp, int x) {
  return *reinterpret_cast<const volatile int *>(comp + x);
}

// A weak load that may be served from this SM's L1 and so be stale.  Used
// where any ancestor of x serves as well as its current parent: comp values
// only ever move to other members of the same tree, and a root stays a root
// until a link hooks it.  Most chases end at the few roots of the largest
// components, whose lines would otherwise be requested from L2 by every warp.
__device__ __forceinline__ int ld_comp_cached(const int *comp, int x) {
  int r;
  asm volatile("ld.global.ca.s32 %0, [%1];" : "=r"(r) : "l"(comp + x));
  return r;
}

// src/cc.cc:40-55 with compare-and-swap on the device.  Reads that may come
// from L1 (stale) are safe here: a stale comp[x] is x itself or one of x's
// ancestors, a vertex that is not a root never becomes one again, and
// comp[high] == low at any time means high and low share a tree for good.
// A value that looks like a root is confirmed from L2 before the
// compare-and-swap, and a failed compare-and-swap returns the current
// parent.  Every pass of the loop moves high strictly up its tree, so the
// loop ends; the iteration limit only guards against a defect.  The roots
// of the large trees are read by almost every warp in the second sampling
// round, which is what keeps those reads in L1.
__device__ void cc_link(int u, int v, int *comp, int *err) {
  int p1 = ld_comp(comp, u);
  int p2 = ld_comp_cached(comp, v);
  // comp[u] == u read fresh: u is a root, so the first pass needs no re-read
  // of its line when u is the higher root (most links of the first round)
  bool u_root = p1 == u;
  for (int it = 0; p1 != p2; it++) {
    if (it >= kChaseLimit) {
      *err = 1;
      return;
    }
    const int high = max(p1, p2), low = min(p1, p2);
    int p_high = (u_root && high == u) ? u : ld_comp_cached(comp, high);
    u_root = false;
    if (p_high == high) {
      p_high = ld_comp(comp, high);
      if (p_high == high) {
        const int old = atomicCAS(comp + high, high, low);
        if (old == high) return;
        p_high = old;
      }
    }
    if (p_high == low) return;
    p1 = ld_comp_cached(comp, p_high);  // at or above high's parent
    p2 = ld_comp_cached(comp, low);
  }
}

struct CcArgs {
  int32_t n, active;
  const int32_t *__restrict__ ooff;
  const int32_t *__restrict__ onbr;
  const int32_t *__restrict__ ioff;  // directed graphs, else null
  const int32_t *__restrict__ inbr;
  const int32_t *__restrict__ perm;
  const int32_t *__restrict__ inv;
  int *comp, *root_min, *second;
  int32_t *out_old;
  GridBarrier *barrier;
  unsigned max_polls;
  int *err;  // page-locked: 1 an iteration limit, 2 a barrier wait ran out
};

// First sampling round (src/cc.cc:100-106): vertex u links with its first
// out-neighbour.  Each thread takes two vertices per pass and loads both
// neighbour ids (random reads of the neighbour array, one HBM sector each)
// before either link, so two such reads are in flight per thread.  The second
// neighbour, mostly in the same sector, is kept for the second round, which
// then reads it in order (62 us a round at Kronecker 2^23 as random reads).
__device__ __forceinline__ void sample_first(const CcArgs &a, int64_t gtid, int64_t stride) {
  for (int64_t u = gtid; u < a.active; u += 2 * stride) {
    const int64_t u2 = u + stride;
    const int s1 = a.ooff[u], e1 = a.ooff[u + 1];
    int s2 = 0, e2 = 0;
    if (u2 < a.active) {
      s2 = a.ooff[u2];
      e2 = a.ooff[u2 + 1];
    }
    const int v1 = s1 < e1 ? a.onbr[s1] : -1;
    const int v2 = s2 < e2 ? a.onbr[s2] : -1;
    const int w1 = s1 + 1 < e1 ? a.onbr[s1 + 1] : -1;
    const int w2 = s2 + 1 < e2 ? a.onbr[s2 + 1] : -1;
    a.second[u] = w1;
    if (u2 < a.active) a.second[u2] = w2;
    if (v1 >= 0) cc_link(static_cast<int>(u), v1, a.comp, a.err);
    if (v2 >= 0) cc_link(static_cast<int>(u2), v2, a.comp, a.err);
  }
}

__device__ __forceinline__ void sample_second(const CcArgs &a, int64_t gtid, int64_t stride) {
  for (int64_t u = gtid; u < a.active; u += stride) {
    const int v = a.second[u];
    if (v >= 0) cc_link(static_cast<int>(u), v, a.comp, a.err);
  }
}

// src/cc.cc:58-66.  No link runs during a compress, so roots are fixed and
// every non-root x has comp[x] != x at all times: c == comp[c] holds exactly
// when c is a root, whether comp[c] was read fresh or from L1.
__device__ __forceinline__ int compress_one(int v, int *comp, int *err) {
  int it = 0;
  int c = ld_comp(comp, v);
  int cc = ld_comp_cached(comp, c);
  while (c != cc) {
    if (++it >= kChaseLimit) {
      *err = 1;
      break;
    }
    comp[v] = cc;
    c = cc;
    cc = ld_comp_cached(comp, c);
  }
  return c;
}

// Final phase: out-neighbours from the third on and, for a directed graph,
// all in-neighbours; vertices of the component of row 0 are skipped
// (src/cc.cc:122-146).  A warp reads the components of 32 consecutive rows at
// once, since nearly all are skipped, then takes the rows left with long lists
// together and the others a lane each (a lane alone would take a microsecond
// an entry, and the other CTAs wait at the barrier for at most some seconds).
__device__ __forceinline__ void link_rest(const CcArgs &a, int giant) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (kThreads / 32);
  for (int64_t b = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5;
       b << 5 < a.active; b += warps) {
    const int u = static_cast<int>(b << 5) + lane;
    const bool left = u < a.active && ld_comp(a.comp, u) != giant;
    // entries of its lists (in- and out-lists of a directed graph differ)
    unsigned entries = 0;
    if (left) {
      entries = a.ooff[u + 1] - a.ooff[u];
      if (a.ioff) entries += a.ioff[u + 1] - a.ioff[u];
    }
    unsigned together = __ballot_sync(0xffffffffu, entries >= kLongList);
    while (together) {
      const int w = static_cast<int>(b << 5) + __ffs(together) - 1;
      together &= together - 1;
      const unsigned oe = a.ooff[w + 1];  // j + 32 may pass 2^31
      for (unsigned j = a.ooff[w] + 2u + lane; j < oe; j += 32)
        cc_link(w, a.onbr[j], a.comp, a.err);
      if (a.ioff) {
        const unsigned ie = a.ioff[w + 1];
        for (unsigned j = a.ioff[w] + static_cast<unsigned>(lane); j < ie; j += 32)
          cc_link(w, a.inbr[j], a.comp, a.err);
      }
      __syncwarp();
    }
    if (left && entries < kLongList) {
      for (int j = a.ooff[u] + 2; j < a.ooff[u + 1]; j++) cc_link(u, a.onbr[j], a.comp, a.err);
      if (a.ioff)
        for (int j = a.ioff[u]; j < a.ioff[u + 1]; j++) cc_link(u, a.inbr[j], a.comp, a.err);
    }
    __syncwarp();
  }
}

// One cooperative launch does a whole run, with a grid barrier between the
// phases (separate launches: 312 us at Kronecker 2^23, 70 us on 1,000
// vertices; 259 and 34 this way).
__global__ void __launch_bounds__(kThreads, kCtasPerSm) cc_kernel(const CcArgs a) {
  __shared__ int s_min[kThreads / 32];
  __shared__ int s_ok;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads;
  const int64_t gtid = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  const int giant = 0;  // the root of row 0's component
  unsigned round = 0;
  auto barrier = [&] {
    const bool ok = grid_barrier(a.barrier, ++round, a.max_polls, &s_ok);
    if (!ok && threadIdx.x == 0) *a.err = 2;
    return ok;
  };
  // roots of the rows [0, active) are rows of [0, active)
  for (int64_t v = gtid; v < a.active; v += stride) {
    a.comp[v] = static_cast<int>(v);
    a.root_min[v] = INT_MAX;
  }
  if (!barrier()) return;
  for (int r = 0; r < 2; r++) {  // neighbor_rounds of src/cc.cc:92
    if (r == 0) sample_first(a, gtid, stride);
    else sample_second(a, gtid, stride);
    if (!barrier()) return;
    for (int64_t v = gtid; v < a.active; v += stride)
      compress_one(static_cast<int>(v), a.comp, a.err);
    if (!barrier()) return;
  }
  link_rest(a, giant);
  if (!barrier()) return;
  // The last compress, fused with the ids mapped back: every vertex chases
  // to its root and offers its original id to the root's minimum.  Members
  // of the component of row 0 (the largest one; half the graph on Kronecker
  // inputs) are reduced per thread and per block first, so its root takes
  // one atomic per block instead of one per vertex.
  int local = INT_MAX;
  for (int64_t v = gtid; v < a.active; v += stride) {
    const int c = compress_one(static_cast<int>(v), a.comp, a.err);
    if (c == giant) local = min(local, a.perm[v]);
    else atomicMin(a.root_min + c, a.perm[v]);
  }
  local = static_cast<int>(__reduce_min_sync(0xffffffffu, static_cast<unsigned>(local)));
  if ((threadIdx.x & 31) == 0) s_min[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int m = static_cast<int>(
        __reduce_min_sync(0xffffffffu, static_cast<unsigned>(s_min[threadIdx.x])));
    if (threadIdx.x == 0 && m != INT_MAX) atomicMin(a.root_min + giant, m);
  }
  if (!barrier()) return;
  // Label of every original id o (a gather, so the writes are coalesced):
  // rows [active, n) have no edges and are their own components.
  for (int64_t o = gtid; o < a.n; o += stride) {
    const int v = a.inv[o];
    a.out_old[o] = v < a.active ? a.root_min[a.comp[v]] : static_cast<int32_t>(o);
  }
  leave_grid(a.barrier);
}

}  // namespace

void FreeCcScratch(CcScratch *c) {
  if (c->mem) cudaFree(c->mem);
  if (c->err) cudaFreeHost(c->err);
  *c = CcScratch();
}

cudaError_t ConnectedComponents(const DeviceGraph &g, CcScratch &cs, cudaStream_t s,
                                unsigned max_polls, int32_t *out_old, std::string *err) {
  const int32_t n = static_cast<int32_t>(g.n);
  cudaError_t e = cudaSuccess;
  if (!cs.comp || cs.cap < n) {
    FreeCcScratch(&cs);
    // one block: the barrier, then the three arrays
    const int64_t cells = (static_cast<int64_t>(n) + 63) & ~int64_t(63);
    e = cudaMalloc(&cs.mem, 256 + 3 * sizeof(int) * cells);
    if (e == cudaSuccess) e = cudaMemsetAsync(cs.mem, 0, sizeof(GridBarrier), s);
    if (e == cudaSuccess)
      e = cudaHostAlloc(reinterpret_cast<void **>(&cs.err), sizeof(int),
                        cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) {
      FreeCcScratch(&cs);
      *err = std::string("connected components: ") + cudaGetErrorString(e);
      return e;
    }
    cs.comp = reinterpret_cast<int *>(static_cast<char *>(cs.mem) + 256);
    cs.root_min = cs.comp + cells;
    cs.second = cs.root_min + cells;
    cs.cap = n;
  }
  CcArgs a;
  a.n = n;
  // Rows without in-neighbours form the tail of the mirror; in an undirected
  // graph they have no edges at all, so no link ever touches them and they
  // stay their own components: the link and compress passes stop before them.
  a.active = g.directed ? n : static_cast<int32_t>(g.bin_row_start[kBinZero]);
  // out-CSR in new ids: the shared CSR of an undirected graph, the
  // renumbered out-CSR of a directed one
  a.ooff = g.directed ? g.orowoff : g.rowoff;
  a.onbr = g.directed ? g.ocol : g.col;
  a.ioff = g.directed ? g.rowoff : nullptr;
  a.inbr = g.directed ? g.col : nullptr;
  a.perm = g.perm;
  a.inv = g.inv;
  a.comp = cs.comp;
  a.root_min = cs.root_min;
  a.second = cs.second;
  a.out_old = out_old;
  a.barrier = static_cast<GridBarrier *>(cs.mem);
  a.max_polls = max_polls;
  a.err = cs.err;
  *cs.err = 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = static_cast<int>(std::max<int64_t>(
      1, std::min<int64_t>((g.n + kThreads - 1) / kThreads, sms * kCtasPerSm)));
  e = LaunchGrid(reinterpret_cast<const void *>(cc_kernel), grid, kThreads, &a, 0, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    *err = std::string("connected components: ") + cudaGetErrorString(e);
    return e;
  }
  if (*cs.err) {
    *err = *cs.err == 1 ? "connected components: link or compress exceeded its iteration limit"
                        : "connected components: a grid barrier ran out of its wait";
    cudaMemsetAsync(cs.mem, 0, sizeof(GridBarrier), s);
    return cudaErrorUnknown;
  }
  return cudaSuccess;
}

}  // namespace prgpu
