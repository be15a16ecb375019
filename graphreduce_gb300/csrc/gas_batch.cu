// gas_batch.cu -- many BFS sources and personalized-PageRank seeds over many
// graphs in one CUDA-graph launch (no reference counterpart).
//
// The graphs are concatenated into one disjoint union graph (vertex ids
// offset per graph), so one device loop serves every instance:
//
//   * multi-source BFS: lane l of a vertex belongs to source l of the
//     vertex's own graph (graphs are disjoint, so lanes of different graphs
//     never meet).  vn[v] = {visited, next}, two 32-bit lane masks in one
//     8-byte record, so a push reads both with one access.  One level
//     pushes every queued vertex's new-lane mask to its out-neighbours
//     (atomicOr, pre-filtered by visited), marking touched vertices in a
//     bitmap; a two-pass compaction over that bitmap writes the level into
//     depth[v][l] for every new lane, folds the lanes into visited and
//     builds the next queue (lane mask, inclusive out-edge ends, CSR offset).
//     Levels with a heavy frontier run bottom-up: every vertex looks for the
//     lanes it lacks in its in-neighbours' frontier masks and stops when it
//     has them.  Depths equal those of one BFS per source.
//   * multi-source SSSP (integer weights, unweighted graphs count 1 per
//     edge): dist[v][l] rows of LS = L rounded up to 4 lanes, cmask[v] the
//     lanes of v that changed in the current iteration.  One bulk-synchronous
//     iteration pushes every queued vertex's changed lanes along its
//     out-edges: the destination's whole row is read once (one 32-byte load
//     for 8 lanes) for all lanes, a lane improves with atomicMin when its
//     candidate is below the value read, and the improved lanes go into
//     cmask and the vertex into the touched bitmap (reductions).  The compaction snapshots
//     each queued vertex's row.  Per lane, distances and iteration counts
//     equal those of one SSSP per source.
//   * multi-seed personalized PageRank, r_l = (1-d) e_{s_l} + d A^T D^-1 r_l
//     for every lane l at once: ranks and contributions are [V][L] rows, so
//     the L lanes of an in-edge's source are one contiguous 4L-byte read.
//     Rows are cut into units of at most 128 in-edges, sorted by length in
//     windows, and the groups of a warp (a thread for one, two or four lanes)
//     walk equally long units side by side with FP32 two-sum compensation,
//     P edges per group and piece (P autotuned); rows of several units leave
//     partials that a second pass folds in a fixed order; a streaming pass
//     turns the rows' sums into ranks, contributions and residuals.  The sums
//     are deterministic.  The loop runs until the largest per-lane L1
//     residual is <= tol.
//
// The loops are WHILE nodes of one CUDA graph (BFS, SSSP, then PPR), each
// preceded by its prologue; a run is one cudaGraphLaunch.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "gas.h"
#include "gas_device.cuh"
#include "gas_engine_impl.h"
#include "gas_internal.h"
#include "gas_sched.h"

using gasdev::kNT;
using gas::fail;

namespace {

inline cudaStream_t S(void *s) { return (cudaStream_t)s; }

constexpr int kMaxLanes = GAS_BATCH_MAX_LANES;

// Device parameters of a run (read by the captured kernels, so that one
// instantiated graph serves any sources, seeds, damping, tolerance and caps).
struct BatchParams {
  double damping;
  double tol;
  int32_t bfs_max_iter;
  int32_t ppr_max_iter;
  int32_t n_sources;  // G * bfs_lanes
  int32_t sssp_max_iter;
  int32_t n_sssp_sources;  // G * sssp_lanes
  int32_t n_seeds;         // G * ppr_lanes
};

__device__ __forceinline__ void set_cond(gas_counters *cnt, bool more, int it,
                                         cudaGraphConditionalHandle h, int in_graph) {
  if (more && it >= cnt->max_iter) cnt->error = GAS_ERR_ITER_CAP;
  cnt->cond = (more && it < cnt->max_iter) ? 1 : 0;
  if (in_graph) cudaGraphSetConditional(h, cnt->cond);
}

__global__ void k_b_reset(gas_counters *cnt, const BatchParams *prm, int which,
                          unsigned long long *edges) {
  cnt->iteration = 0;
  cnt->error = 0;
  cnt->cond = 0;
  cnt->n_changed = 0;
  cnt->n_scatter_edges = 0;
  cnt->mode = 0;
  cnt->max_iter = which == 0 ? prm->bfs_max_iter
                 : which == 1 ? prm->ppr_max_iter : prm->sssp_max_iter;
  if (edges) *edges = 0ull;
}

// ---------------------------------------------------------------------------
// multi-source BFS
// ---------------------------------------------------------------------------
struct MsPushPol {
  typedef int32_t Val;
  static constexpr bool kMapNeedsVertex = false;
  const int32_t *csr_dst;
  const int32_t *q_mask;
  uint32_t *vn;  // [V][2]: visited, next
  uint32_t *tbits;
  __device__ Val zero() const { return 0; }
  __device__ Val reduce(Val a, Val) const { return a; }
  __device__ Val map(int, int, int) const { return 0; }
  __device__ void emit(int, int, Val) const {}
  // a: queue position of the pushing vertex, pos: CSR position of the edge.
  // visited does not change during the push; next[v] starts the push at 0
  // and only gains bits, so lanes already seen in it (a plain, possibly
  // stale load) need no atomic; every thread that adds lanes also marks v
  // as touched (both reductions, no thread waits for a result).
  __device__ __forceinline__ void visit(int a, int, int pos) const {
    const int v = __ldg(csr_dst + pos);
    const uint2 p = reinterpret_cast<const uint2 *>(vn)[v];
    const uint32_t m = (uint32_t)__ldg(q_mask + a) & ~p.x;
    if (m && (p.y & m) != m) {
      atomicOr(vn + 2 * (size_t)v + 1, m);  // fire-and-forget; the touched bit is idempotent
      atomicOr(tbits + ((uint32_t)v >> 5), 1u << (v & 31));
    }
  }
};

enum { kModePush = 0, kModePull = 1 };

// Level 0: every (graph, lane) source.
__global__ void k_ms_seed(const int32_t *src_global, const BatchParams *prm, int L,
                          uint32_t *vn, uint32_t *tbits) {
  const int n = prm->n_sources;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = src_global[i];
    if (v < 0) continue;
    atomicOr(vn + 2 * (size_t)v + 1, 1u << (i % L));
    atomicOr(tbits + ((uint32_t)v >> 5), 1u << (v & 31));
  }
}

// The direction of the next level (Beamer, Asanovic & Patterson, SC'12, with
// edges counted once per lane): bottom-up once the new frontier's lane-edges
// exceed 1/kMsAlpha of those not yet explored, top-down again when the
// frontier shrinks below V / kMsBeta vertices.  alpha: on R-MAT and
// Erdos-Renyi graphs with 2 to 32 lanes every level with a ratio of 0.25 or
// more reads fewer edges bottom-up (0.02 to 0.7 E against 0.4 to 1.0 E), every
// one at 0.08 or less more.
// A wrong bottom-up level costs more than a wrong top-down one (16 lanes on
// 5 R-MAT graphs of 30 edges per vertex: 1.02 ms with alpha 6, 0.43 with 3,
// 0.53 top-down only); 16 R-MAT graphs, 16 lanes: 0.66 ms with 3 to 8, 1.08
// top-down only.
constexpr int kMsAlpha = 3;
constexpr int kMsBeta = 24;
struct MsDir {
  unsigned long long frontier;  // lane-edges of the new frontier (summed by the count pass)
  unsigned long long explored;  // of every frontier so far
};

// One bottom-up level: a thread per vertex looks, among its in-neighbours,
// for the lanes it still lacks in the frontier's lane masks fr[], and stops
// when it has them all.  Only lanes alive in its graph (with a frontier) are
// looked for, so a source in a small component costs nothing once it is
// done.  The first in-edge alone (sources are in id order, low ids are the
// hubs), then four at a time; a row unfinished after 29 in-edges is taken
// over by its whole warp, 128 at a time, or one thread would walk a hub's
// row alone.  Writes the new lanes and whole words of the touched bitmap, as
// the push leaves them, without an atomic.
struct MsPull {
  const int32_t *csc_off, *csc_src;
  const uint32_t *fr, *alive;
  const int32_t *g_off;
  int G, nV;
};

__device__ __forceinline__ void ms_pull(const MsPull &a, uint32_t *vn, uint32_t *tbits) {
  const int32_t *csc_off = a.csc_off, *csc_src = a.csc_src, *g_off = a.g_off;
  const uint32_t *fr = a.fr, *alive = a.alive;
  const int G = a.G, nV = a.nV;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kAlone = 29;
  const int lane = threadIdx.x & 31;
  const int nW = (nV + 31) / 32;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w < nW; w += nwarps) {
    // the graph of the word's first vertex: the last one starting at or before it
    int g = 0;
    for (int lo = 0, hi = G - 1; lo < hi;) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(g_off + mid) <= w * 32)
        lo = mid;
      else
        hi = mid - 1;
      g = lo;
    }
    const int v = w * 32 + lane;
    uint32_t want = 0u, found = 0u;
    int i = 0, end = 0;
    if (v < nV) {
      while (v >= __ldg(g_off + g + 1)) ++g;
      want = __ldg(alive + g) & ~vn[2 * (size_t)v];
      if (want) {
        i = __ldg(csc_off + v);
        end = __ldg(csc_off + v + 1);
      }
    }
    const int stop = end - i > kAlone ? i + kAlone : end;
    if (i < end) found = __ldg(fr + __ldg(csc_src + i)) & want;
    for (++i; i < stop && found != want; i += 4) {
      int u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = i + j < stop ? __ldg(csc_src + i + j) : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j) found |= u[j] >= 0 ? __ldg(fr + u[j]) & want : 0u;
    }
    for (unsigned rest = __ballot_sync(FULL, found != want && stop < end); rest;
         rest &= rest - 1) {
      const int l = __ffs(rest) - 1;
      const uint32_t lw = __shfl_sync(FULL, want, l);
      const int le = __shfl_sync(FULL, end, l);
      uint32_t lf = __shfl_sync(FULL, found, l);
      for (int p = __shfl_sync(FULL, stop, l); p < le && lf != lw; p += 128) {
        int u[4];
        uint32_t f = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int q = p + 32 * j + lane;
          u[j] = q < le ? __ldg(csc_src + q) : -1;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) f |= u[j] >= 0 ? __ldg(fr + u[j]) : 0u;
        lf |= __reduce_or_sync(FULL, f) & lw;
      }
      if (lane == l) found = lf;
    }
    if (found) vn[2 * (size_t)v + 1] = found;
    const unsigned t = __ballot_sync(FULL, found != 0u);
    if (lane == 0 && t) tbits[w] = t;
  }
}

// One level in the direction the spine chose (one kernel: a node less per
// level than a push and a pull of which one returns at once).
__global__ void __launch_bounds__(kNT)
    k_ms_level(MsPushPol pol, gasdev::SlabSource src, MsPull pull, const gas_counters *cnt) {
  if (cnt->mode == kModePull)
    ms_pull(pull, pol.vn, pol.tbits);
  else
    gasdev::slab_loop<MsPushPol, false>(pol, src, nullptr, nullptr, nullptr, nullptr, nullptr);
}

// The touched-vertex traversal shared by the two compaction passes: a warp
// owns a run of WW words of the touched bitmap (lanes 0..WW-1 load them) and
// walks it in rounds of up to 8 words, skipping a round whose words are all
// clear; lane l takes vertex 32 w + l of each word, and a round's loads are
// issued before any is used.  For a touched vertex: its new lanes and
// out-edge range.  The count pass keeps each warp's totals, so the write
// passes take their offsets without counting again.  WW is 16 on large
// unions and less where that would leave fewer than four blocks per SM
// (ms_words): 16 BFS lanes on 50 K vertices, 13 blocks of 16-word runs,
// spent a fifth of the run in this pass.
constexpr int kMsWarps = kNT / 32;

template <int WW>
struct MsRound {
  static constexpr int R = WW < 8 ? WW : 8;
  uint32_t nw[R];  // new lanes (0: not touched or nothing new)
  int off[R];
  int deg[R];
};

// The lane's word of the warp's run (lanes 0..WW-1; 0 past the bitmap).
template <int WW>
__device__ __forceinline__ uint32_t ms_word(const uint32_t *tbits, int nW, int w0) {
  const int lane = threadIdx.x & 31;
  return lane < WW && w0 + lane < nW ? tbits[w0 + lane] : 0u;
}

template <int WW>
__device__ __forceinline__ bool ms_round_live(unsigned nz, int r) {
  return ((nz >> r) & ((1u << MsRound<WW>::R) - 1u)) != 0u;
}

// Round r (words w0 + r .. ).  next: the SSSP's changed-lane words; vn (BFS,
// next unused): the {visited, next} pairs, new lanes = next & ~visited.
template <int WW>
__device__ __forceinline__ void ms_round_load(uint32_t myword, const uint32_t *next,
                                              const uint32_t *vn, const int32_t *csr_off,
                                              int w0, int r, MsRound<WW> &m) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < MsRound<WW>::R; ++i) {
    const uint32_t word = __shfl_sync(0xffffffffu, myword, r + i);
    m.nw[i] = 0u;
    m.off[i] = 0;
    m.deg[i] = 0;
    if ((word >> lane) & 1u) {
      const int v = (w0 + r + i) * 32 + lane;
      if (vn) {
        const uint2 p = reinterpret_cast<const uint2 *>(vn)[v];
        m.nw[i] = p.y & ~p.x;
      } else {
        m.nw[i] = next[v];
      }
      m.off[i] = csr_off[v];
      m.deg[i] = csr_off[v + 1] - m.off[i];
    }
  }
}

// Pass 1: per block (queue entries, out-edges) for the spine and per warp
// for the write pass; with lanes_active, also the OR of the new lanes of the
// queue's entries (the SSSP loop).
template <int WW>
__global__ void __launch_bounds__(kNT)
    k_ms_count(const uint32_t *tbits, const uint32_t *next, const uint32_t *vn,
               const int32_t *csr_off, int nW, int32_t *part, int2 *wpart,
               uint32_t *lanes_active, MsDir *dir) {
  __shared__ unsigned long long s_m[kMsWarps];
  __shared__ int s_q[kMsWarps], s_d[kMsWarps];
  __shared__ uint32_t s_l[kMsWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * kMsWarps + warp) * WW;
  const uint32_t myword = ms_word<WW>(tbits, nW, w0);
  const unsigned nz = __ballot_sync(0xffffffffu, myword != 0u);
  int q = 0, d = 0;
  unsigned long long le = 0ull;  // out-edges times new lanes
  uint32_t lanes = 0u;
#pragma unroll 1
  for (int r = 0; r < WW; r += MsRound<WW>::R) {
    if (!ms_round_live<WW>(nz, r)) continue;  // warp-uniform
    MsRound<WW> m;
    ms_round_load<WW>(myword, next, vn, csr_off, w0, r, m);
#pragma unroll
    for (int i = 0; i < MsRound<WW>::R; ++i) {
      const bool in = m.nw[i] && m.deg[i] > 0;
      q += in;
      d += in ? m.deg[i] : 0;
      le += (unsigned long long)m.deg[i] * __popc(m.nw[i]);
      if (m.deg[i] > 0) lanes |= m.nw[i];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    q += __shfl_xor_sync(0xffffffffu, q, o);
    d += __shfl_xor_sync(0xffffffffu, d, o);
    lanes |= __shfl_xor_sync(0xffffffffu, lanes, o);
    le += __shfl_xor_sync(0xffffffffu, le, o);
  }
  if (lane == 0) {
    s_m[warp] = le;
    s_q[warp] = q;
    s_d[warp] = d;
    s_l[warp] = lanes;
    wpart[blockIdx.x * kMsWarps + warp] = make_int2(q, d);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int tq = 0, td = 0;
    uint32_t tl = 0u;
    for (int k = 0; k < kMsWarps; ++k) {
      tq += s_q[k];
      td += s_d[k];
      tl |= s_l[k];
    }
    part[2 * blockIdx.x] = tq;
    part[2 * blockIdx.x + 1] = td;
    if (lanes_active && tl) atomicOr(lanes_active, tl);
    if (dir) {
      unsigned long long tm = 0ull;
      for (int k = 0; k < kMsWarps; ++k) tm += s_m[k];
      if (tm) atomicAdd(&dir->frontier, tm);
    }
  }
}

// The warp's first queue entry and out-edge offset: its block's (scanned by
// the spine) plus the totals of the block's earlier warps.
__device__ __forceinline__ int2 ms_warp_base(const int32_t *part, const int2 *wpart,
                                             int warp) {
  int2 b = make_int2(part[2 * blockIdx.x], part[2 * blockIdx.x + 1]);
  for (int k = 0; k < warp; ++k) {
    const int2 t = wpart[blockIdx.x * kMsWarps + k];
    b.x += t.x;
    b.y += t.y;
  }
  return b;
}

// The new lanes' depths of a word's 32 vertices (nw per lane, `live` their
// ballot): the warp walks the rows 32 / G at a time, lane by lane, so that a
// row's lanes leave in one store (a thread storing its own row's lanes one by
// one wrote a sector per depth: 118 us for 13 M depths, 49 now).
__device__ __forceinline__ void ms_store_depths(int32_t *depth, int L, int G, int v0, uint32_t nw,
                                                unsigned live, int level) {
  const int lane = threadIdx.x & 31;
  const int rows = 32 / G, l = lane % G, sub = lane / G;
  for (int r = 0; r < 32; r += rows) {
    if (!((live >> r) & (rows == 32 ? 0xffffffffu : (1u << rows) - 1u))) continue;  // uniform
    const uint32_t m = __shfl_sync(0xffffffffu, nw, r + sub);
    if ((m >> l) & 1u) depth[(size_t)(v0 + r + sub) * L + l] = level;
  }
}

// Pass 2: depths of the new lanes (level = the iteration the spine just
// counted) and visited; for a top-down next level the queue and the push's
// chunk partition at the chunk size the spine chose, for a bottom-up one
// every vertex's frontier mask and the graphs' alive lanes; clears next and
// the touched bitmap.
template <int WW>
__global__ void __launch_bounds__(kNT, 5)
    k_ms_write(uint32_t *tbits, uint32_t *vn, const int32_t *csr_off,
               int nW, const int32_t *part, const int2 *wpart, int L, int G,
               const gas_counters *cnt, int32_t *depth, int32_t *q_mask, int32_t *q_end,
               int32_t *q_delta, int32_t *chunk_row, uint32_t *fr, uint32_t *alive, const int32_t *g_off,
               int n_graphs, int nV) {
  // rows spanning many chunks (hubs), written by the whole warp at the end
  constexpr int kBig = 64;
  __shared__ int3 s_big[kMsWarps][kBig];
  __shared__ int s_nbig[kMsWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * kMsWarps + warp) * WW;
  const uint32_t myword = ms_word<WW>(tbits, nW, w0);
  const unsigned nz = __ballot_sync(0xffffffffu, myword != 0u);
  const int level = cnt->iteration;
  if (myword) tbits[w0 + lane] = 0u;
  if (cnt->mode == kModePull) {  // grid-uniform
    int g = 0;  // of the run's first vertex; the graphs are in vertex order
    for (int lo = 0, hi = n_graphs - 1; lo < hi;) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(g_off + mid) <= w0 * 32)
        lo = mid;
      else
        hi = mid - 1;
      g = lo;
    }
    constexpr int R = MsRound<WW>::R;
#pragma unroll 1
    for (int r = 0; r < WW; r += R) {
      uint32_t nws[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const uint32_t word = __shfl_sync(0xffffffffu, myword, r + i);
        const int v = (w0 + r + i) * 32 + lane;
        nws[i] = 0u;
        if ((word >> lane) & 1u) {
          const uint2 p = reinterpret_cast<const uint2 *>(vn)[v];
          nws[i] = p.y & ~p.x;
          reinterpret_cast<uint2 *>(vn)[v] = make_uint2(p.x | nws[i], 0u);
        }
        if (v < nV) fr[v] = nws[i];
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const uint32_t nw = nws[i];
        const int v = (w0 + r + i) * 32 + lane;
        const unsigned live = __ballot_sync(0xffffffffu, nw != 0u);
        if (!live) continue;  // warp-uniform
        ms_store_depths(depth, L, G, (w0 + r + i) * 32, nw, live, level);
        int gv = g;
        if (nw)
          while (v >= __ldg(g_off + gv + 1)) ++gv;
        const int g0 = __shfl_sync(0xffffffffu, gv, __ffs(live) - 1);
        if (__all_sync(0xffffffffu, !nw || gv == g0)) {
          const uint32_t all = __reduce_or_sync(0xffffffffu, nw);
          if (lane == 0 && (__ldcg(alive + g0) & all) != all) atomicOr(alive + g0, all);
        } else if (nw) {
          atomicOr(alive + gv, nw);
        }
        g = g0;
      }
    }
    return;
  }
  if (!nz) return;  // warp-uniform: nothing touched in the run
  const int cl = cnt->push_chunk_log2;
  if (lane == 0) s_nbig[warp] = 0;
  __syncwarp();
  const int2 base = ms_warp_base(part, wpart, warp);
  int bq = base.x, bd = base.y;
#pragma unroll 1
  for (int r = 0; r < WW; r += MsRound<WW>::R) {
    if (!ms_round_live<WW>(nz, r)) continue;  // warp-uniform
    MsRound<WW> m;
    ms_round_load<WW>(myword, nullptr, vn, csr_off, w0, r, m);
#pragma unroll
    for (int i = 0; i < MsRound<WW>::R; ++i) {
      const int v = (w0 + r + i) * 32 + lane;
      const uint32_t word = __shfl_sync(0xffffffffu, myword, r + i);
      if (!word) continue;  // warp-uniform
      const bool touched = (word >> lane) & 1u;
      const uint32_t nw = m.nw[i];
      if (touched) vn[2 * (size_t)v + 1] = 0u;
      if (nw) vn[2 * (size_t)v] |= nw;
      const unsigned live = __ballot_sync(0xffffffffu, nw != 0u);
      if (!live) continue;  // warp-uniform
      ms_store_depths(depth, L, G, (w0 + r + i) * 32, nw, live, level);
      const int deg = nw ? m.deg[i] : 0;
      const unsigned qb = __ballot_sync(0xffffffffu, deg > 0);
      if (!qb) continue;
      int incl = deg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (deg > 0) {
        const int pos = bq + __popc(qb & ((1u << lane) - 1u));
        const int end = bd + incl;
        q_mask[pos] = (int32_t)nw;
        q_end[pos] = end;
        q_delta[pos] = m.off[i] - (end - deg);
        // chunk partition of the next push (chunks starting in this range)
        const int c0 = (end - deg + (1 << cl) - 1) >> cl, c1 = (end + (1 << cl) - 1) >> cl;
        int slot = kBig;
        if (c1 - c0 > 4) slot = atomicAdd(&s_nbig[warp], 1);
        if (slot < kBig)
          s_big[warp][slot] = make_int3(pos, c0, c1);
        else
          for (int c = c0; c < c1; ++c) chunk_row[c] = pos;
      }
      bq += __popc(qb);
      bd += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncwarp();
  const int nbig = min(s_nbig[warp], kBig);
  for (int k = 0; k < nbig; ++k) {
    const int3 rr = s_big[warp][k];
    for (int c = rr.y + lane; c < rr.z; c += 32) chunk_row[c] = rr.x;
  }
}

// ---------------------------------------------------------------------------
// multi-source SSSP
// ---------------------------------------------------------------------------
constexpr int32_t kSsspInf = INT_MAX - 100000;  // the SSSP Program's gatherZero

struct MssPushPol {
  typedef int32_t Val;
  static constexpr bool kMapNeedsVertex = false;
  const int32_t *csr_dst;
  const int32_t *csr_w;   // null: every edge weighs 1
  const int32_t *q_mask;  // [queue] lanes that changed
  const int32_t *q_vals;  // [queue][LS] row at the end of the last iteration
  int32_t *dist;          // [V][LS]
  uint32_t *cmask;        // [V] lanes changed in this iteration
  uint32_t *tbits;
  int LS;
  __device__ Val zero() const { return 0; }
  __device__ Val reduce(Val a, Val) const { return a; }
  __device__ Val map(int, int, int) const { return 0; }
  __device__ void emit(int, int, Val) const {}
  // The row read is a plain load: a value it returns was held by the lane
  // during this iteration, so a candidate below it lowers the lane's final
  // value under its start value (the lane changed) and a candidate at or
  // above it cannot lower the final value.
  __device__ __forceinline__ void visit(int a, int, int pos) const {
    const int v = __ldg(csr_dst + pos);
    const long long w = csr_w ? __ldg(csr_w + pos) : 1;
    const uint32_t m = (uint32_t)__ldg(q_mask + a);
    const int4 *cur4 = reinterpret_cast<const int4 *>(dist + (size_t)v * LS);
    const int4 *qv4 = reinterpret_cast<const int4 *>(q_vals + (size_t)a * LS);
    int32_t *row = dist + (size_t)v * LS;
    uint32_t nb = 0u;
    for (int c = 0; c < (LS >> 2); ++c) {
      const uint32_t mc = (m >> (4 * c)) & 0xFu;
      if (!mc) continue;
      const int4 cu = cur4[c];
      const int4 qv = __ldg(qv4 + c);
      const int cur[4] = {cu.x, cu.y, cu.z, cu.w};
      const int val[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!((mc >> k) & 1u)) continue;
        const long long cl = (long long)val[k] + w;
        const int cand = cl > kSsspInf ? kSsspInf : (int)cl;
        if (cand < cur[k]) {
          atomicMin(row + 4 * c + k, cand);
          nb |= 1u << (4 * c + k);
        }
      }
    }
    if (nb && (cmask[v] & nb) != nb) {
      atomicOr(cmask + v, nb);  // reductions: the touched bit is idempotent
      atomicOr(tbits + ((uint32_t)v >> 5), 1u << (v & 31));
    }
  }
};

// 32-byte row loads (one instruction, one sector): the row must be 32-byte
// aligned.  row8 is a plain load (the row changes during the push), nc8 a
// read-only one.
__device__ __forceinline__ void row8(const int32_t *p, int (&r)[8]) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "l"(p));
}
__device__ __forceinline__ void nc8(const int32_t *p, int (&r)[8]) {
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "l"(p));
}

// Rows of at most 8 lanes (NC = 1 or 2 16-byte chunks): the same push split
// into probe (the edge's loads and the destination row) and commit, so that
// both slabs' row reads are in flight before either slab's updates.  Every
// lane of the row is tried, not only the changed ones: a lane of u that did
// not change in the last iteration already pushed its value along this edge
// when it last changed, so its candidate is at or above the destination's
// value at the start of this iteration (and of any value read during it)
// and changes nothing.  Weights are at most 100000, as the SSSP Program's
// gatherZero assumes, so val + w does not overflow.
template <int NC>
struct MssPushPolStaged {
  typedef int32_t Val;
  static constexpr bool kMapNeedsVertex = false;
  const int32_t *csr_dst;
  const int32_t *csr_w;
  const int32_t *q_vals;
  int32_t *dist;
  uint32_t *cmask;
  uint32_t *tbits;
  __device__ Val zero() const { return 0; }
  __device__ Val reduce(Val a, Val) const { return a; }
  __device__ Val map(int, int, int) const { return 0; }
  __device__ void emit(int, int, Val) const {}
  struct Probe {
    int v, w, a;  // v < 0: no edge
    int cur[4 * NC];
  };
  __device__ __forceinline__ Probe probe(bool valid, int a, int, int pos) const {
    Probe p;
    p.v = -1;
    p.w = 0;
    p.a = a;
    if (valid) {
      p.v = __ldg(csr_dst + pos);
      p.w = csr_w ? __ldg(csr_w + pos) : 1;
      const int32_t *r = dist + (size_t)p.v * (4 * NC);
      if constexpr (NC == 2) {
        row8(r, p.cur);
      } else {
        const int4 c4 = *reinterpret_cast<const int4 *>(r);
        p.cur[0] = c4.x;
        p.cur[1] = c4.y;
        p.cur[2] = c4.z;
        p.cur[3] = c4.w;
      }
    }
    return p;
  }
  __device__ __forceinline__ void commit(const Probe &p) const {
    if (p.v < 0) return;
    const int32_t *q = q_vals + (size_t)p.a * (4 * NC);
    int val[4 * NC];
    if constexpr (NC == 2) {
      nc8(q, val);
    } else {
      const int4 q4 = __ldg(reinterpret_cast<const int4 *>(q));
      val[0] = q4.x;
      val[1] = q4.y;
      val[2] = q4.z;
      val[3] = q4.w;
    }
    int32_t *row = dist + (size_t)p.v * (4 * NC);
    uint32_t nb = 0u;
#pragma unroll
    for (int k = 0; k < 4 * NC; ++k) {
      const int cand = min(val[k] + p.w, kSsspInf);
      if (cand < p.cur[k]) {
        atomicMin(row + k, cand);
        nb |= 1u << k;
      }
    }
    // the lanes and the touched bit as fire-and-forget reductions (both are
    // idempotent, so no thread waits for an atomic's result); issued
    // without first loading cmask[v] to skip repeats: that dependent load
    // cost more than the repeated reductions (8 lanes at R-MAT scale 22:
    // 0.406 -> 0.370 ms per push)
    if (nb) {
      atomicOr(cmask + p.v, nb);
      atomicOr(tbits + ((uint32_t)p.v >> 5), 1u << (p.v & 31));
    }
  }
};

template <class Pol>
__global__ void __launch_bounds__(kNT) k_mss_push(Pol pol, gasdev::SlabSource src) {
  gasdev::slab_loop<Pol, false>(pol, src, nullptr, nullptr, nullptr, nullptr, nullptr);
}

__global__ void k_mss_init(int32_t *dist, size_t n, uint32_t *lanes_active,
                           int32_t *lane_rounds) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x)
    dist[k] = kSsspInf;
  if (blockIdx.x == 0 && threadIdx.x < kMaxLanes) {
    lane_rounds[threadIdx.x] = 0;
    if (threadIdx.x == 0) *lanes_active = 0u;
  }
}

// Iteration 0: every (graph, lane) source gets distance 0 and is changed.
__global__ void k_mss_seed(const int32_t *src_global, const BatchParams *prm, int L, int LS,
                           int32_t *dist, uint32_t *cmask, uint32_t *tbits) {
  const int n = prm->n_sssp_sources;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = src_global[i];
    if (v < 0) continue;
    dist[(size_t)v * LS + i % L] = 0;
    atomicOr(cmask + v, 1u << (i % L));
    atomicOr(tbits + ((uint32_t)v >> 5), 1u << (v & 31));
  }
}

// Pass 2 of the compaction: the next queue (snapshot row, inclusive
// out-edge ends, CSR offset; the changed lanes for rows wider than 8 lanes)
// and the push's chunk partition at the chunk size the spine chose; clears
// cmask and the touched bitmap.
template <int WW>
__global__ void __launch_bounds__(kNT, 4)
    k_mss_write(uint32_t *tbits, uint32_t *cmask, const int32_t *csr_off, int nW,
                const int32_t *part, const int2 *wpart, int LS, const int32_t *dist,
                int32_t *q_mask, int32_t *q_vals, int32_t *q_end, int32_t *q_delta,
                int32_t *chunk_row, const gas_counters *cnt) {
  // rows spanning many chunks (hubs), written by the whole warp at the end
  constexpr int kBig = 64;
  __shared__ int3 s_big[kMsWarps][kBig];
  __shared__ int s_nbig[kMsWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * kMsWarps + warp) * WW;
  const uint32_t myword = ms_word<WW>(tbits, nW, w0);
  const unsigned nz = __ballot_sync(0xffffffffu, myword != 0u);
  if (!nz) return;  // warp-uniform: nothing touched in the run
  const int cl = cnt->push_chunk_log2;
  if (lane == 0) s_nbig[warp] = 0;
  __syncwarp();
  const int2 base = ms_warp_base(part, wpart, warp);
  int bq = base.x, bd = base.y;
  if (myword) tbits[w0 + lane] = 0u;
#pragma unroll 1
  for (int r = 0; r < WW; r += MsRound<WW>::R) {
    if (!ms_round_live<WW>(nz, r)) continue;  // warp-uniform
    MsRound<WW> m;
    ms_round_load<WW>(myword, cmask, nullptr, csr_off, w0, r, m);
#pragma unroll
    for (int i = 0; i < MsRound<WW>::R; ++i) {
      const int v = (w0 + r + i) * 32 + lane;
      const uint32_t word = __shfl_sync(0xffffffffu, myword, r + i);
      if (!word) continue;  // warp-uniform
      if ((word >> lane) & 1u) cmask[v] = 0u;
      const uint32_t nw = m.nw[i];
      const int deg = nw ? m.deg[i] : 0;
      const unsigned qb = __ballot_sync(0xffffffffu, deg > 0);
      if (!qb) continue;
      int incl = deg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (deg > 0) {
        const int pos = bq + __popc(qb & ((1u << lane) - 1u));
        const int end = bd + incl;
        if (LS > 8) q_mask[pos] = (int32_t)nw;  // rows of up to 8 lanes try every lane
        q_end[pos] = end;
        q_delta[pos] = m.off[i] - (end - deg);
        const int4 *src4 = reinterpret_cast<const int4 *>(dist + (size_t)v * LS);
        int4 *dst4 = reinterpret_cast<int4 *>(q_vals + (size_t)pos * LS);
        for (int c = 0; c < (LS >> 2); ++c) dst4[c] = src4[c];
        const int c0 = (end - deg + (1 << cl) - 1) >> cl, c1 = (end + (1 << cl) - 1) >> cl;
        int slot = kBig;
        if (c1 - c0 > 4) slot = atomicAdd(&s_nbig[warp], 1);
        if (slot < kBig)
          s_big[warp][slot] = make_int3(pos, c0, c1);
        else
          for (int c = c0; c < c1; ++c) chunk_row[c] = pos;
      }
      bq += __popc(qb);
      bd += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncwarp();
  const int nbig = min(s_nbig[warp], kBig);
  for (int k = 0; k < nbig; ++k) {
    const int3 rr = s_big[warp][k];
    for (int c = rr.y + lane; c < rr.z; c += 32) chunk_row[c] = rr.x;
  }
}

// Exclusive scan of the block pairs in one pass (1024 threads, each holding a
// run of ceil(nb / 1024) pairs in registers), then the loop control of the
// BFS and SSSP loops: queue totals, the push's chunk size (512 edges per
// warp, halved down to 64 while there would be fewer than two chunks per
// push warp), the lanes of the new queue (each has one more push to run;
// SSSP only), the WHILE condition.
constexpr int kMssSpineNT = 1024;
constexpr int kMssSpineRegs = 8;

__global__ void __launch_bounds__(kMssSpineNT)
    k_mss_spine(int2 *part, int nb, gas_counters *cnt, int push_warps,
                unsigned long long *edges, uint32_t *lanes_active, int32_t *lane_rounds,
                MsDir *dir, uint32_t *alive, int G, unsigned long long lane_edges, int nV,
                cudaGraphConditionalHandle h, int in_graph, int first) {
  if (alive)  // gathered again by the write pass
    for (int g = threadIdx.x; g < G; g += kMssSpineNT) alive[g] = 0u;
  const int per = (nb + kMssSpineNT - 1) / kMssSpineNT;
  const int b0 = threadIdx.x * per, b1 = min(nb, b0 + per);
  const bool in_regs = per <= kMssSpineRegs;
  int2 x[kMssSpineRegs];
  int sq = 0, sd = 0;
  if (in_regs) {
#pragma unroll
    for (int k = 0; k < kMssSpineRegs; ++k) x[k] = b0 + k < b1 ? part[b0 + k] : make_int2(0, 0);
#pragma unroll
    for (int k = 0; k < kMssSpineRegs; ++k) {
      sq += x[k].x;
      sd += x[k].y;
    }
  } else {
    for (int b = b0; b < b1; ++b) {
      sq += part[b].x;
      sd += part[b].y;
    }
  }
  __shared__ int2 s_w[kMssSpineNT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int iq = sq, id = sd;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int oq = __shfl_up_sync(0xffffffffu, iq, d);
    const int od = __shfl_up_sync(0xffffffffu, id, d);
    if (lane >= d) {
      iq += oq;
      id += od;
    }
  }
  if (lane == 31) s_w[warp] = make_int2(iq, id);
  __syncthreads();
  int pq = iq - sq, pd = id - sd, tq = 0, td = 0;
#pragma unroll 8
  for (int k = 0; k < kMssSpineNT / 32; ++k) {
    const int2 t = s_w[k];
    if (k < warp) {
      pq += t.x;
      pd += t.y;
    }
    tq += t.x;
    td += t.y;
  }
  if (in_regs) {
#pragma unroll
    for (int k = 0; k < kMssSpineRegs; ++k) {
      if (b0 + k < b1) {
        part[b0 + k] = make_int2(pq, pd);
        pq += x[k].x;
        pd += x[k].y;
      }
    }
  } else {
    for (int b = b0; b < b1; ++b) {
      const int2 y = part[b];
      part[b] = make_int2(pq, pd);
      pq += y.x;
      pd += y.y;
    }
  }
  if (threadIdx.x == 0) {
    cnt->n_changed = tq;
    cnt->n_scatter_edges = td;
    int cl = gasdev::kSlabChunkLog2;
    while (cl > gasdev::kSlabChunkMinLog2 && (td >> cl) < 2 * push_warps) --cl;
    cnt->push_chunk_log2 = cl;
    if (lanes_active) {
      const uint32_t la = *lanes_active;
      *lanes_active = 0u;
      for (int l = 0; l < kMaxLanes; ++l)
        if ((la >> l) & 1u) ++lane_rounds[l];
    }
    if (dir) {  // BFS: the next level's direction
      const unsigned long long f = dir->frontier, seen = (first ? 0ull : dir->explored) + f;
      const bool pulling = !first && cnt->mode == kModePull;
      const bool pull = pulling ? (long long)tq * kMsBeta > nV
                                : f * kMsAlpha > (lane_edges > seen ? lane_edges - seen : 0ull);
      cnt->mode = pull && td > 0 ? kModePull : kModePush;
      dir->explored = seen;
      dir->frontier = 0ull;
    }
    const int it = first ? 0 : ++cnt->iteration;
    set_cond(cnt, td > 0, it, h, in_graph);
    if (cnt->cond) *edges += (unsigned long long)td;
  }
}

// ---------------------------------------------------------------------------
// multi-seed personalized PageRank
// ---------------------------------------------------------------------------
struct __align__(8) CVal {
  float s, c;
};

// Knuth two-sum: a + b = s + c exactly.
__device__ __forceinline__ CVal two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  return CVal{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp))};
}

// Compensations add up in c.
__device__ __forceinline__ CVal two_sum_add(CVal a, CVal b) {
  const CVal t = two_sum(a.s, b.s);
  return CVal{t.s, __fadd_rn(__fadd_rn(a.c, b.c), t.c)};
}

struct PprArgs {
  const int32_t *csc_off, *csr_off;
  const int32_t *ne_vid;  // the rows with in-edges
  // the plan (below): sources in walking order, the slices' first steps, the
  // units' destinations, the pieces' first slices, the rows of several units
  // and their first partials
  const int32_t *idx, *step_off, *unit_dst, *piece_start, *long_row, *long_slot;
  int32_t n_pieces, n_long, L, G, n_ne, nV;
  CVal *partial;      // [slots][L] partial sums of the units of long rows
  float *sum;         // [n_ne][L] the rows' sums of an iteration
  float *rank, *contrib;  // [V][L], [V + 1][L]: the last row stays 0
  const uint32_t *seed_mask;
  const BatchParams *prm;
  gas_counters *cnt;
  double *l1_part;        // [blocks][G] of k_ppr_rows
  double *lane_resid;
  unsigned int *ticket;   // blocks of k_ppr_rows done (left at 0)
};

// The gather's plan.  A row's in-edges are cut into units of at most 128 edges;
// the units of a window of 2,048 are sorted by their number of steps (8 edges
// each), and S units that follow one another in that order, S the groups of a
// warp, form a slice: the warp walks them side by side, and since they are
// (nearly) equally long their rows end at the same step.  The sources are
// stored step by step, S x 8 to a step, short units padded with the index of a
// contribution row of zeros: a warp's reads of them are whole lines and need no
// bounds.  Whole steps of padding come first, so that all units of a slice end
// in its last step, the one summed term by term.  (A walk of consecutive rows
// by 8 groups finds a row end in three of four steps, in one group, and all
// wait for it: 630 us per iteration at 64 M edges and 16 lanes, issue slots
// half busy with 16 warps per SM, against 367.)
constexpr int kPprU = 8;          // in-edges of a step of the gather
constexpr int kPprUnit = 128;     // in-edges of a unit
constexpr int kPprWindow = 2048;  // units sorted together
constexpr int kPprLong = 16;      // rows of more units are folded by a whole CTA

// VL consecutive lanes of a row, one load or store.
template <int VL>
struct Lanes {
  float f[VL];
};

template <int VL>
__device__ __forceinline__ Lanes<VL> ppr_ld(const float *p) {
  Lanes<VL> o;
  if constexpr (VL == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    o.f[0] = t.x; o.f[1] = t.y; o.f[2] = t.z; o.f[3] = t.w;
  } else if constexpr (VL == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
    o.f[0] = t.x; o.f[1] = t.y;
  } else {
    o.f[0] = __ldg(p);
  }
  return o;
}

template <int VL>
__device__ __forceinline__ void ppr_st(float *p, const Lanes<VL> &v) {
  if constexpr (VL == 4)
    *reinterpret_cast<float4 *>(p) = make_float4(v.f[0], v.f[1], v.f[2], v.f[3]);
  else if constexpr (VL == 2)
    *reinterpret_cast<float2 *>(p) = make_float2(v.f[0], v.f[1]);
  else
    *p = v.f[0];
}

template <int VL>
__device__ __forceinline__ void ppr_contrib8(const PprArgs &a, const int (&u)[kPprU], int l,
                                             Lanes<VL> (&x)[kPprU]) {
#pragma unroll
  for (int j = 0; j < kPprU; ++j) x[j] = ppr_ld<VL>(a.contrib + (size_t)u[j] * a.L + l);
}

// The gather: a warp takes a piece of consecutive slices, a group of G / VL
// threads (VL lanes each) a unit of each, with the next step's contribution
// rows and two steps' sources in flight.  A step is summed pairwise in FP32
// (relative error <= 3 u of the step's sum, the terms being non-negative),
// the last step of a slice term by term; both go into the unit's sum by
// two-sum, so a row's error stays near 3 u of its value.  Rows of one unit
// store their sum (by row, no dependent load), units of longer rows leave
// partials for k_ppr_fix.  What follows a row's sum (rank, contribution,
// residual) is k_ppr_rows', a streaming pass: done here, each row end
// stalled the walk on four loads.
template <int VL>
__global__ void __launch_bounds__(kNT) k_ppr_units(PprArgs a) {
  const int T = a.G / VL, S = 32 / T;
  const int lane = threadIdx.x & 31, g = lane / T;
  const int l = lane % T * VL;
  const bool on = l < a.L;
  const int lc = on ? l : 0;
  const int nwarps = (int)((gridDim.x * kNT) >> 5);
  for (int k = (int)((blockIdx.x * kNT + threadIdx.x) >> 5); k < a.n_pieces; k += nwarps) {
    int s = __ldg(a.piece_start + k);
    const int s_end = __ldg(a.piece_start + k + 1);
    if (s == s_end) continue;  // warp-uniform
    int t = __ldg(a.step_off + s);
    const int t_end = __ldg(a.step_off + s_end);
    int next = __ldg(a.step_off + s + 1), next2 = 0;
    int dst = __ldg(a.unit_dst + (size_t)s * S + g), dst2 = 0;
    if (s + 1 < s_end) {
      next2 = __ldg(a.step_off + s + 2);
      dst2 = __ldg(a.unit_dst + (size_t)(s + 1) * S + g);
    }
    const int32_t *p = a.idx + ((size_t)t * S + g) * kPprU;
    int u[kPprU], u2[kPprU];
    Lanes<VL> x[kPprU], y[kPprU];
    nc8(p, u);
    if (t + 1 < t_end) nc8(p + S * kPprU, u2);
    ppr_contrib8<VL>(a, u, lc, x);
    CVal acc[VL];
#pragma unroll
    for (int q = 0; q < VL; ++q) acc[q] = CVal{0.f, 0.f};
    for (;;) {
      const bool more = t + 1 < t_end;
      if (more) {
#pragma unroll
        for (int j = 0; j < kPprU; ++j) u[j] = u2[j];
        if (t + 2 < t_end) nc8(p + 2 * S * kPprU, u2);
        ppr_contrib8<VL>(a, u, lc, y);
      }
      if (t + 1 < next) {  // warp-uniform
#pragma unroll
        for (int q = 0; q < VL; ++q) {
          const float h = __fadd_rn(
              __fadd_rn(__fadd_rn(x[0].f[q], x[1].f[q]), __fadd_rn(x[2].f[q], x[3].f[q])),
              __fadd_rn(__fadd_rn(x[4].f[q], x[5].f[q]), __fadd_rn(x[6].f[q], x[7].f[q])));
          acc[q] = two_sum_add(acc[q], CVal{h, 0.f});
        }
      } else {
#pragma unroll
        for (int j = 0; j < kPprU; ++j)
#pragma unroll
          for (int q = 0; q < VL; ++q) acc[q] = two_sum_add(acc[q], CVal{x[j].f[q], 0.f});
        if (on && dst >= 0) {
          Lanes<VL> o;
#pragma unroll
          for (int q = 0; q < VL; ++q) o.f[q] = __fadd_rn(acc[q].s, acc[q].c);
          ppr_st<VL>(a.sum + (size_t)dst * a.L + l, o);
        } else if (on && dst != INT_MIN) {
#pragma unroll
          for (int q = 0; q < VL; ++q) a.partial[(size_t)~dst * a.L + l + q] = acc[q];
        }
#pragma unroll
        for (int q = 0; q < VL; ++q) acc[q] = CVal{0.f, 0.f};
        ++s;
        next = next2;
        dst = dst2;
        if (s + 1 < s_end) {
          next2 = __ldg(a.step_off + s + 2);
          dst2 = __ldg(a.unit_dst + (size_t)(s + 1) * S + g);
        }
      }
      if (!more) break;
#pragma unroll
      for (int j = 0; j < kPprU; ++j) x[j] = y[j];
      ++t;
      p += S * kPprU;
    }
  }
}

// VL lanes' partials, 16 bytes at a time.
template <int VL>
struct Partials {
  CVal p[VL];
};

template <int VL>
__device__ __forceinline__ Partials<VL> ppr_partials(const CVal *p) {
  Partials<VL> o;
  if constexpr (VL >= 2) {
#pragma unroll
    for (int q = 0; q < VL; q += 2) {
      const float4 t = *reinterpret_cast<const float4 *>(p + q);
      o.p[q] = CVal{t.x, t.y};
      o.p[q + 1] = CVal{t.z, t.w};
    }
  } else {
    o.p[0] = *p;
  }
  return o;
}

// Rows of several units, their partials folded in a fixed order: a group per
// row, or the whole CTA (every group a strided share, then the groups' sums)
// for rows of more than kPprLong units -- one group folding a hub's 1,200
// partials one after the other took 90 us.  Rows next to one another go to
// different CTAs: hubs have neighbouring ids, and a CTA folds its hubs one
// after the other.
template <int VL>
__global__ void __launch_bounds__(kNT) k_ppr_fix(PprArgs a) {
  __shared__ Partials<VL> s_part[kNT];
  __shared__ int s_end[kNT];
  const int T = a.G / VL;
  const int l = threadIdx.x % T * VL, g = threadIdx.x / T, groups = kNT / T;
  const bool on = l < a.L;
  for (int k0 = blockIdx.x; k0 < a.n_long; k0 += gridDim.x * groups) {
    const int k = k0 + g * gridDim.x;
    int r = -1, b = 0, e = 0;
    if (k < a.n_long) {
      r = __ldg(a.long_row + k);
      b = __ldg(a.long_slot + k);
      e = __ldg(a.long_slot + k + 1);
    }
    const bool lng = e - b > kPprLong;
    Partials<VL> acc, next;
#pragma unroll
    for (int i = 0; i < VL; ++i) acc.p[i] = CVal{0.f, 0.f};
    if (r >= 0 && !lng && on) {
#pragma unroll 2
      for (int q = b; q < e; ++q) {
        next = ppr_partials<VL>(a.partial + (size_t)q * a.L + l);
#pragma unroll
        for (int i = 0; i < VL; ++i) acc.p[i] = two_sum_add(acc.p[i], next.p[i]);
      }
      Lanes<VL> o;
#pragma unroll
      for (int i = 0; i < VL; ++i) o.f[i] = __fadd_rn(acc.p[i].s, acc.p[i].c);
      ppr_st<VL>(a.sum + (size_t)r * a.L + l, o);
    }
    if (!__syncthreads_or(lng)) continue;  // CTA-uniform
    if (l == 0) s_end[g] = lng ? e : -1;
    __syncthreads();
    for (int h = 0; h < groups; ++h) {
      const int he = s_end[h];
      if (he < 0) continue;  // CTA-uniform
      const int kh = k0 + h * gridDim.x;
      const int hb = __ldg(a.long_slot + kh);
#pragma unroll
      for (int i = 0; i < VL; ++i) acc.p[i] = CVal{0.f, 0.f};
      if (on)
#pragma unroll 4
        for (int q = hb + g; q < he; q += groups) {
          next = ppr_partials<VL>(a.partial + (size_t)q * a.L + l);
#pragma unroll
          for (int i = 0; i < VL; ++i) acc.p[i] = two_sum_add(acc.p[i], next.p[i]);
        }
      s_part[threadIdx.x] = acc;
      __syncthreads();
      for (int w = groups >> 1; w > 0; w >>= 1) {
        if (g < w) {
#pragma unroll
          for (int i = 0; i < VL; ++i)
            s_part[threadIdx.x].p[i] =
                two_sum_add(s_part[threadIdx.x].p[i], s_part[threadIdx.x + w * T].p[i]);
        }
        __syncthreads();
      }
      if (g == 0 && on) {
        Lanes<VL> o;
#pragma unroll
        for (int i = 0; i < VL; ++i)
          o.f[i] = __fadd_rn(s_part[threadIdx.x].p[i].s, s_part[threadIdx.x].p[i].c);
        ppr_st<VL>(a.sum + (size_t)__ldg(a.long_row + kh) * a.L + l, o);
      }
      __syncthreads();
    }
  }
}

// A row's inputs, loaded before any is used; then its new rank and
// contribution from its sum, and its L1 step.
template <int VL>
struct PprRow {
  int v, deg;
  uint32_t seed;
  Lanes<VL> sum, old;
};

template <int VL>
__device__ __forceinline__ void ppr_row_load(const PprArgs &a, int l, PprRow<VL> &w) {
  w.seed = __ldg(a.seed_mask + w.v);
  w.deg = __ldg(a.csr_off + w.v + 1) - __ldg(a.csr_off + w.v);
  const float *o = a.rank + (size_t)w.v * a.L + l;
  if constexpr (VL == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(o);
    w.old.f[0] = t.x; w.old.f[1] = t.y; w.old.f[2] = t.z; w.old.f[3] = t.w;
  } else {
#pragma unroll
    for (int q = 0; q < VL; ++q) w.old.f[q] = o[q];
  }
}

// A thread's sum of L1 steps, in no fewer bits than FP64 sums have but (nearly)
// without FP64 (two conversions and two additions per rank took three quarters
// of k_ppr_rows' time at GB300's FP64 rate).  A step |new - old| = s + c exactly
// (two-sum); s goes into a, what that addition rounds off and c into b, what
// those round off into t.  N steps are off by at most N^3 2^-73 of their sum,
// FP64 by up to N 2^-53, so every kL1Flush rows go into an FP64 sum.  (34 M
// ranks, 2.1 M vertices of 16 lanes: 528 us per iteration of all kernels, with
// FP64 throughout 649; with a and b alone, whose additions round at 2^-49, 524.)
constexpr int kL1Flush = 64;
struct L1Sum {
  float a = 0.f, b = 0.f, t = 0.f;
  __device__ __forceinline__ void add(CVal step) {
    if (step.s < 0.f) step = CVal{-step.s, -step.c};
    const CVal x = two_sum(a, step.s), y = two_sum(b, step.c), z = two_sum(y.s, x.c);
    a = x.s;
    b = z.s;
    t = __fadd_rn(t, __fadd_rn(y.c, z.c));
  }
  __device__ __forceinline__ double value() const {
    return __dadd_rn((double)a, __dadd_rn((double)b, (double)t));
  }
};

template <int VL>
__device__ __forceinline__ void ppr_row_finish(const PprArgs &a, int l, const PprRow<VL> &w,
                                               float d, float base, L1Sum (&l1)[VL]) {
  Lanes<VL> rank, contrib;
#pragma unroll
  for (int q = 0; q < VL; ++q) {
    const float b = ((w.seed >> (l + q)) & 1u) ? base : 0.f;
    const float r = __fadd_rn(b, __fmul_rn(d, w.sum.f[q]));
    l1[q].add(two_sum(r, -w.old.f[q]));
    rank.f[q] = r;
    contrib.f[q] = w.deg ? __fdiv_rn(r, (float)w.deg) : 0.f;
  }
  ppr_st<VL>(a.rank + (size_t)w.v * a.L + l, rank);
  ppr_st<VL>(a.contrib + (size_t)w.v * a.L + l, contrib);
}

// Ranks, contributions and residual of every row with in-edges; in the first
// iteration also of those without (their rank is (1-d) [seed] from then on,
// so they are skipped afterwards).  Bound by memory: four arrays of [V][L]
// floats streamed, two rows per group in flight.  The last block done adds
// the blocks' residuals up, in a fixed order, and sets the loop condition:
// on while the largest lane's is above tol.
template <int VL>
__global__ void __launch_bounds__(kNT)
    k_ppr_rows(PprArgs a, cudaGraphConditionalHandle h, int in_graph) {
  const int T = a.G / VL;
  const int l = threadIdx.x % T * VL, grp = threadIdx.x / T, per_block = kNT / T;
  const float d = (float)a.prm->damping, base = (float)(1.0 - a.prm->damping);
  const bool first = a.cnt->iteration == 0;
  L1Sum l1[VL];
  double done[VL];  // of the rows already flushed
#pragma unroll
  for (int q = 0; q < VL; ++q) done[q] = 0.0;
  int rows = 0;
  const auto flush = [&](int n) {
    rows += n;
    if (rows < kL1Flush) return;
    rows = 0;
#pragma unroll
    for (int q = 0; q < VL; ++q) {
      done[q] = __dadd_rn(done[q], l1[q].value());
      l1[q] = L1Sum();
    }
  };
  if (l < a.L) {
    const int stride = gridDim.x * per_block;
    int i = blockIdx.x * per_block + grp;
    for (; i < a.n_ne - stride; i += 2 * stride) {  // (n_ne + stride may not fit an int)
      PprRow<VL> w[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        w[k].v = __ldg(a.ne_vid + i + k * stride);
        w[k].sum = ppr_ld<VL>(a.sum + (size_t)(i + k * stride) * a.L + l);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) ppr_row_load<VL>(a, l, w[k]);
#pragma unroll
      for (int k = 0; k < 2; ++k) ppr_row_finish<VL>(a, l, w[k], d, base, l1);
      flush(2);
    }
    if (i < a.n_ne) {
      PprRow<VL> w;
      w.v = __ldg(a.ne_vid + i);
      w.sum = ppr_ld<VL>(a.sum + (size_t)i * a.L + l);
      ppr_row_load<VL>(a, l, w);
      ppr_row_finish<VL>(a, l, w, d, base, l1);
    }
    if (first)
      for (int v = blockIdx.x * per_block + grp; v < a.nV; v += stride)
        if (__ldg(a.csc_off + v) == __ldg(a.csc_off + v + 1)) {
          PprRow<VL> w;
          w.v = v;
#pragma unroll
          for (int q = 0; q < VL; ++q) w.sum.f[q] = 0.f;
          ppr_row_load<VL>(a, l, w);
          ppr_row_finish<VL>(a, l, w, d, base, l1);
          flush(1);
        }
  }
  // per-lane block sums in a fixed order
  __shared__ double s[kNT * VL];
#pragma unroll
  for (int q = 0; q < VL; ++q) s[grp * a.G + l + q] = __dadd_rn(done[q], l1[q].value());
  __syncthreads();
  if (threadIdx.x < a.G) {
    double t = 0.0;
    for (int j = threadIdx.x; j < kNT * VL; j += a.G) t += s[j];
    a.l1_part[(size_t)blockIdx.x * a.G + threadIdx.x] = t;
  }
  const int g = threadIdx.x / a.G, groups = kNT / a.G;
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double v = 0.0;
#pragma unroll 8
  for (int b = g; b < (int)gridDim.x; b += groups)
    v += __ldcg(a.l1_part + (size_t)b * a.G + threadIdx.x % a.G);
  s[threadIdx.x] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < a.G)
    for (int q = 0; q < groups; ++q) t += s[q * a.G + threadIdx.x];
  __syncthreads();
  if (threadIdx.x < a.G) s[threadIdx.x] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double mx = 0.0;
    for (int q = 0; q < a.L; ++q) {
      a.lane_resid[1 + q] = s[q];
      mx = s[q] > mx ? s[q] : mx;
    }
    a.lane_resid[0] = mx;
    *a.ticket = 0u;
    const int it = ++a.cnt->iteration;
    set_cond(a.cnt, !(mx <= a.prm->tol), it, h, in_graph);
  }
}

// The plan's kernels, in order.  Units of each row, and the rows of several.
__global__ void k_plan_count(const int32_t *ne_end, int n_ne, int32_t *units, int32_t *slots,
                             int32_t *longs) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= n_ne; r += gridDim.x * blockDim.x) {
    int n = 0;
    if (r < n_ne) n = (ne_end[r] - (r > 0 ? ne_end[r - 1] : 0) + kPprUnit - 1) / kPprUnit;
    units[r] = n;
    slots[r] = n > 1 ? n : 0;
    longs[r] = n > 1 ? 1 : 0;
  }
}

// (After scans of the three.)  The units' rows; the long rows.
__global__ void k_plan_units(const int32_t *units, const int32_t *slots, const int32_t *longs,
                             int n_ne, int32_t *unit_row, int32_t *long_row, int32_t *long_slot) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= n_ne; r += gridDim.x * blockDim.x) {
    if (r == n_ne) {
      long_slot[longs[r]] = slots[r];
      break;
    }
    const int b = units[r], e = units[r + 1];
    for (int u = b; u < e; ++u) unit_row[u] = r;
    if (e - b > 1) {
      long_row[longs[r]] = r;
      long_slot[longs[r]] = slots[r];
    }
  }
}

// A window's units in order of their steps (stable): (first edge, edges) and
// destination of every place.
__global__ void __launch_bounds__(kNT)
    k_plan_sort(const int32_t *ne_end, const int32_t *units, const int32_t *slots,
                const int32_t *unit_row, int U, int2 *place, int32_t *unit_dst) {
  constexpr int kSteps = kPprUnit / kPprU;   // 1 .. 16
  constexpr int kItems = kPprWindow / kNT;   // consecutive units of a thread
  __shared__ int cnt[kSteps][kNT];
  __shared__ int tot[kSteps];
  const int t = threadIdx.x, u0 = blockIdx.x * kPprWindow;
  int2 at[kItems];
  int dst[kItems], key[kItems];
#pragma unroll
  for (int j = 0; j < kSteps; ++j) cnt[j][t] = 0;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int u = u0 + t * kItems + i;
    key[i] = -1;
    if (u < U) {
      const int r = unit_row[u], c = u - units[r], n = units[r + 1] - units[r];
      const int e0 = (r > 0 ? ne_end[r - 1] : 0) + c * kPprUnit;
      const int len = min(kPprUnit, ne_end[r] - e0);
      at[i] = make_int2(e0, len);
      dst[i] = n == 1 ? r : ~(slots[r] + c);
      key[i] = (len + kPprU - 1) / kPprU - 1;
      ++cnt[key[i]][t];
    }
  }
  __syncthreads();
  // exclusive scan in (key, thread) order: a warp scans two keys
  const int lane = t & 31, warp = t >> 5;
  for (int k = warp; k < kSteps; k += kNT / 32) {
    int run = 0;
    for (int b = 0; b < kNT; b += 32) {
      const int x = cnt[k][b + lane];
      int incl = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
      }
      cnt[k][b + lane] = run + incl - x;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tot[k] = run;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    if (key[i] < 0) continue;
    int pos = u0 + cnt[key[i]][t]++;
    for (int k = 0; k < key[i]; ++k) pos += tot[k];
    place[pos] = at[i];
    unit_dst[pos] = dst[i];
  }
}

// Steps of every slice of S units (the longest's).
__global__ void k_plan_steps(const int2 *place, int U, int S, int n_slices, int32_t *step_off) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s <= n_slices;
       s += gridDim.x * blockDim.x) {
    int m = 0;
    if (s < n_slices)
      for (int g = 0; g < S && s * S + g < U; ++g) m = max(m, place[s * S + g].y);
    step_off[s] = (m + kPprU - 1) / kPprU;
  }
}

// (After a scan of the steps.)  The sources in walking order, a warp per
// slice; places past the last unit have no destination.
__global__ void __launch_bounds__(kNT)
    k_plan_index(const int2 *place, const int32_t *step_off, const int32_t *csc_src, int U, int S,
                 int n_slices, int nV, int32_t *idx, int32_t *unit_dst) {
  const int lane = threadIdx.x & 31, nwarps = (int)((gridDim.x * kNT) >> 5);
  for (int s = (int)((blockIdx.x * kNT + threadIdx.x) >> 5); s < n_slices; s += nwarps) {
    const int t0 = step_off[s], t1 = step_off[s + 1];
    const int n = (t1 - t0) * S * kPprU;
    for (int i = lane; i < n; i += 32) {
      const int step = i / (S * kPprU), g = i / kPprU % S, j = i % kPprU;
      int v = nV;
      if (s * S + g < U) {
        const int2 p = place[s * S + g];
        const int lead = t1 - t0 - (p.y + kPprU - 1) / kPprU;
        const int e = (step - lead) * kPprU + j;
        if (e >= 0 && e < p.y) v = csc_src[p.x + e];
      }
      idx[(size_t)t0 * S * kPprU + i] = v;
    }
    if (lane < S && s * S + lane >= U) unit_dst[s * S + lane] = INT_MIN;
  }
}

// The first slice of every piece of `steps` steps.
__global__ void k_plan_pieces(const int32_t *step_off, int n_slices, int n_pieces, int steps,
                              int32_t *piece_start) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k <= n_pieces;
       k += gridDim.x * blockDim.x) {
    const long long want = (long long)k * steps;
    int lo = 0, hi = n_slices;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (step_off[mid] < want)
        lo = mid + 1;
      else
        hi = mid;
    }
    piece_start[k] = lo;
  }
}

// Each (graph, lane) seed's bit.
__global__ void k_ppr_seed(const int32_t *seeds, const BatchParams *prm, int L,
                           uint32_t *seed_mask) {
  const int n = prm->n_seeds;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (seeds[i] >= 0) atomicOr(seed_mask + seeds[i], 1u << (i % L));
}

// r0 = e_seed per lane; contributions accordingly.
__global__ void k_ppr_init(const uint32_t *seed_mask, const int32_t *csr_off, int nV, int L,
                           float *rank, float *contrib) {
  const size_t n = (size_t)nV * L;
  if (blockIdx.x == 0 && threadIdx.x < L) contrib[n + threadIdx.x] = 0.f;  // the plan's padding
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const int v = (int)(k / L), l = (int)(k % L);
    const float r = ((seed_mask[v] >> l) & 1u) ? 1.f : 0.f;
    float c = 0.f;
    if (r != 0.f) {
      const int deg = csr_off[v + 1] - csr_off[v];
      c = deg ? __fdiv_rn(r, (float)deg) : 0.f;
    }
    rank[k] = r;
    contrib[k] = c;
  }
}

__global__ void k_ppr_precond(gas_counters *cnt, cudaGraphConditionalHandle h, int in_graph) {
  set_cond(cnt, true, 0, h, in_graph);
}

}  // namespace

// ---------------------------------------------------------------------------
// The batch object.
// ---------------------------------------------------------------------------
struct gas_batch {
  std::vector<int32_t> v_off{0};  // first vertex of every graph; back() = V
  std::vector<int32_t> src, dst;  // union edge list (global ids) until built
  std::vector<int32_t> w;         // its weights, once a weighted graph came
  bool weighted = false;
  int64_t n_edges = 0;
  gas_engine *eng = nullptr;      // holds the union graph (CSR + CSC)
  bool built = false;
  gas_counters *cnt = nullptr;    // [3] device: BFS loop, PPR loop, SSSP loop
  gas_counters *h_cnt = nullptr;  // [3] pinned
  BatchParams *prm = nullptr;     // device
  unsigned long long *edges = nullptr;  // BFS edges pushed
  double *resid = nullptr;        // [1 + 32] max and per-lane PPR residual
  // BFS
  uint32_t *vn = nullptr, *next = nullptr, *tbits = nullptr;  // vn: [V][2] BFS pairs
  int32_t *depth = nullptr, *q_mask = nullptr, *q_end = nullptr,
          *q_delta = nullptr, *part = nullptr, *qpart = nullptr, *srcs = nullptr;
  int32_t depth_lanes = 0, srcs_cap = 0;
  // bottom-up levels: frontier masks [V], alive lanes [graphs], the graphs'
  // first vertices, the direction rule's sums
  uint32_t *fr = nullptr, *alive = nullptr;
  int32_t *g_off = nullptr;
  MsDir *dir = nullptr;
  // SSSP (shares the frontier arrays above; next is the changed-lane mask)
  int32_t *dist = nullptr, *q_vals = nullptr, *sssp_srcs = nullptr, *lane_rounds = nullptr;
  uint32_t *lanes_active = nullptr;
  unsigned long long *sssp_edges = nullptr;
  int32_t dist_ls = 0, sssp_srcs_cap = 0;
  // the arrays above and below by what allocates them: the frontier, the SSSP
  // rows, the BFS state, the PPR rows and plan
  DeviceGroup frontier_mem, dist_mem, bfs_mem, ppr_mem, plan_mem, piece_mem;
  // profiling of the SSSP pushes (direct launches, events around each push)
  bool profiling = false;
  cudaEvent_t pev[2] = {nullptr, nullptr};
  gas_kernel_profile prof{};
  // PPR
  // the gather's plan (plan_mem), for slices of plan_S units, and its pieces
  // (piece_mem) of piece_edges edges per group
  int32_t *pp_idx = nullptr, *pp_step_off = nullptr, *pp_unit_dst = nullptr,
          *pp_long_row = nullptr, *pp_long_slot = nullptr, *pp_piece_start = nullptr;
  CVal *partial = nullptr;
  int32_t plan_S = 0, n_slices = 0, n_steps = 0, n_long = 0, n_slots = 0;
  float *rank = nullptr, *contrib = nullptr, *sum = nullptr;
  uint32_t *seed_mask = nullptr;
  int32_t *seeds = nullptr;
  double *l1 = nullptr;
  unsigned int *ticket = nullptr;
  int32_t n_pieces = 0, piece_edges = 0, ppr_lanes = 0, l1_cap = 0, seeds_cap = 0;
  int32_t tuned_piece = 0;
  // cached graph
  cudaGraphExec_t graph = nullptr;
  int32_t g_bfs_lanes = -1, g_ppr_lanes = -1, g_piece = -1, g_sssp_lanes = -1;
};

namespace {

template <class T>
void bfree(T *&p) {
  if (p) cudaFree((void *)p);
  p = nullptr;
}

// Another allocation in place of p's.  On failure p is null (the caller's size
// of it has to say so) and the runtime's last error is cleared, or the next
// launch would report it.
template <class T>
cudaError_t renew(T *&p, size_t bytes) {
  bfree(p);
  const cudaError_t ce = cudaMalloc((void **)&p, bytes);
  if (ce != cudaSuccess) {
    p = nullptr;
    cudaGetLastError();
  }
  return ce;
}

void drop_graph(gas_batch *b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  b->graph = nullptr;
  b->g_bfs_lanes = b->g_ppr_lanes = b->g_piece = b->g_sssp_lanes = -1;
}

void free_state(gas_batch *b) {
  drop_graph(b);
  b->frontier_mem.free();
  b->dist_mem.free();
  b->bfs_mem.free();
  b->ppr_mem.free();
  b->plan_mem.free();
  b->piece_mem.free();
  bfree(b->depth); bfree(b->srcs);
  bfree(b->seed_mask); bfree(b->seeds); bfree(b->l1); bfree(b->ticket);
  bfree(b->sssp_srcs); bfree(b->lane_rounds);
  bfree(b->lanes_active);
  b->dist_ls = b->sssp_srcs_cap = 0;
  b->n_pieces = b->piece_edges = b->ppr_lanes = b->depth_lanes = b->plan_S = 0;
  b->srcs_cap = b->l1_cap = b->seeds_cap = 0;
}

// Lanes per thread of the PPR kernels: four (16-byte loads) from 12 lanes up,
// two below, where a warp of 16 or 32 groups has too few rows in flight per
// register (per run, 1 / 2 / 4 lanes a thread: 16 lanes - / 11.7 / 9.9 ms, 8
// lanes - / 3.1 / 3.5, 4 lanes - / 2.2 / 2.6).  Two lanes go one to a thread.
int ppr_vl(int L) { return L % 4 == 0 && L > 8 ? 4 : L % 2 == 0 && L > 2 ? 2 : 1; }

int lane_group(int L) {
  int g = 1;
  while (g < L) g <<= 1;
  return g;
}

int nwords(const gas_batch *b) { return (b->eng->nV + 31) / 32; }
// Bitmap words per warp of the compaction passes.
int ms_words(const gas_batch *b) {
  const int64_t room = 4LL * b->eng->num_sms * kMsWarps;  // warps of four blocks per SM
  return nwords(b) <= 2 * room ? 2 : nwords(b) <= 4 * room ? 4 : 16;
}
int ms_blocks(const gas_batch *b) {
  const int words = ms_words(b) * kMsWarps;
  return std::max(1, (nwords(b) + words - 1) / words);
}
// qpart: the blocks' (entries, out-edges) pairs, one spare pair, then the
// blocks' per-warp pairs
int2 *ms_wpart(const gas_batch *b) {
  return reinterpret_cast<int2 *>(b->qpart + 2 * ((size_t)ms_blocks(b) + 1));
}

// The frontier arrays the BFS and SSSP loops share (they run one after the
// other, each prologue resetting them).
gas_status_t ensure_frontier(gas_batch *b) {
  gas_engine *e = b->eng;
  const size_t nV = std::max(1, e->nV), nW = std::max(1, nwords(b));
  if (!b->next) {
    // part: the SSSP push cuts its queue's edges into chunks of 64 to 512 edges
    CUDA_TRY(b->frontier_mem.alloc(
        {GROUP_PART(b->next, nV * 4), GROUP_PART(b->tbits, nW * 4), GROUP_PART(b->q_mask, nV * 4),
         GROUP_PART(b->q_end, nV * 4), GROUP_PART(b->q_delta, nV * 4),
         GROUP_PART(b->part, (((size_t)e->nE >> gasdev::kSlabChunkMinLog2) + 2) * 4),
         GROUP_PART(b->qpart,
                    2 * ((size_t)ms_blocks(b) + 1 + (size_t)ms_blocks(b) * kMsWarps) * 4)}));
  }
  return GAS_OK;
}

gas_status_t ensure_sssp(gas_batch *b, int lanes, int n_sources) {
  gas_engine *e = b->eng;
  const size_t nV = std::max(1, e->nV);
  GAS_TRY(ensure_frontier(b));
  const int LS = (lanes + 3) & ~3;
  if (b->dist_ls != LS) {
    drop_graph(b);
    b->dist_ls = 0;
    CUDA_TRY(b->dist_mem.alloc(
        {GROUP_PART(b->dist, nV * LS * 4), GROUP_PART(b->q_vals, nV * LS * 4)}));
    b->dist_ls = LS;
  }
  if (!b->lane_rounds) CUDA_TRY(renew(b->lane_rounds, kMaxLanes * 4));
  if (!b->lanes_active) CUDA_TRY(renew(b->lanes_active, 4));
  if (b->sssp_srcs_cap < n_sources) {
    drop_graph(b);
    b->sssp_srcs_cap = 0;
    CUDA_TRY(renew(b->sssp_srcs, (size_t)std::max(1, n_sources) * 4));
    b->sssp_srcs_cap = n_sources;
  }
  return GAS_OK;
}

// s: the run's stream, which the initial values are ordered by (they are in
// place at return: the state outlives a run that fails, and its stream).
gas_status_t ensure_bfs(gas_batch *b, int lanes, int n_sources, cudaStream_t s) {
  gas_engine *e = b->eng;
  const size_t nV = std::max(1, e->nV);
  GAS_TRY(ensure_frontier(b));
  if (!b->vn) {
    const size_t ng = b->v_off.size();
    CUDA_TRY(b->bfs_mem.alloc({GROUP_PART(b->vn, nV * 8), GROUP_PART(b->fr, nV * 4),
                               GROUP_PART(b->alive, ng * 4), GROUP_PART(b->g_off, ng * 4),
                               GROUP_PART(b->dir, sizeof(MsDir))}));
    CUDA_TRY(cudaMemcpyAsync(b->g_off, b->v_off.data(), b->v_off.size() * 4,
                             cudaMemcpyHostToDevice, s));
    CUDA_TRY(cudaMemsetAsync(b->dir, 0, sizeof(MsDir), s));
    CUDA_TRY(cudaStreamSynchronize(s));
  }
  if (b->depth_lanes != lanes) {
    drop_graph(b);
    b->depth_lanes = 0;
    CUDA_TRY(renew(b->depth, nV * lanes * 4));
    b->depth_lanes = lanes;
  }
  if (b->srcs_cap < n_sources) {
    drop_graph(b);
    b->srcs_cap = 0;
    CUDA_TRY(renew(b->srcs, (size_t)std::max(1, n_sources) * 4));
    b->srcs_cap = n_sources;
  }
  return GAS_OK;
}

// The gather's plan for slices of S units; reads three counts back, so it
// waits for the stream.
gas_status_t build_ppr_plan(gas_batch *b, int S, cudaStream_t s) {
  gas_engine *e = b->eng;
  const int n_ne = e->n_ne, grid = 8 * e->num_sms;
  b->plan_S = 0;
  b->plan_mem.free();
  DeviceGroup tmp, tmp2;
  struct Guard {
    DeviceGroup &a, &b;
    ~Guard() { a.free(); b.free(); }
  } guard{tmp, tmp2};
  int32_t *units = nullptr, *slots = nullptr, *longs = nullptr, *part = nullptr;
  CUDA_TRY(tmp.alloc({GROUP_PART(units, ((size_t)n_ne + 1) * 4),
                      GROUP_PART(slots, ((size_t)n_ne + 1) * 4),
                      GROUP_PART(longs, ((size_t)n_ne + 1) * 4),
                      GROUP_PART(part, (size_t)gas::device_scan_parts(n_ne + 1) * 4)}));
  k_plan_count<<<grid, 256, 0, s>>>(e->ne_end, n_ne, units, slots, longs);
  CUDA_TRY(cudaGetLastError());
  int32_t total[3];  // units, partial slots, long rows
  int32_t *scanned[3] = {units, slots, longs};
  for (int i = 0; i < 3; ++i) {
    GAS_TRY(gas::device_scan_excl(scanned[i], n_ne + 1, part, s));
    CUDA_TRY(cudaMemcpyAsync(&total[i], scanned[i] + n_ne, 4, cudaMemcpyDeviceToHost, s));
  }
  CUDA_TRY(cudaStreamSynchronize(s));
  const int U = total[0], n_slices = (int)(((long long)U + S - 1) / S);
  int32_t *unit_row = nullptr, *spart = nullptr, *steps = nullptr;
  int2 *place = nullptr;
  CUDA_TRY(tmp2.alloc({GROUP_PART(unit_row, (size_t)U * 4), GROUP_PART(place, (size_t)U * 8),
                       GROUP_PART(steps, ((size_t)n_slices + 1) * 4),
                       GROUP_PART(spart, (size_t)gas::device_scan_parts(n_slices + 1) * 4)}));
  // the destinations are made with the places and the number of steps known
  // after them: two groups, the long rows with the first
  int32_t *unit_dst = nullptr, *long_row = nullptr, *long_slot = nullptr;
  DeviceGroup dests;
  struct Guard1 {
    DeviceGroup &a;
    ~Guard1() { a.free(); }
  } guard1{dests};
  CUDA_TRY(dests.alloc({GROUP_PART(unit_dst, (size_t)n_slices * S * 4),
                        GROUP_PART(long_row, (size_t)total[2] * 4),
                        GROUP_PART(long_slot, ((size_t)total[2] + 1) * 4)}));
  k_plan_units<<<grid, 256, 0, s>>>(units, slots, longs, n_ne, unit_row, long_row, long_slot);
  if (U > 0)
    k_plan_sort<<<(U + kPprWindow - 1) / kPprWindow, kNT, 0, s>>>(e->ne_end, units, slots,
                                                                unit_row, U, place, unit_dst);
  k_plan_steps<<<grid, 256, 0, s>>>(place, U, S, n_slices, steps);
  CUDA_TRY(cudaGetLastError());
  GAS_TRY(gas::device_scan_excl(steps, n_slices + 1, spart, s));
  int32_t n_steps = 0;
  CUDA_TRY(cudaMemcpyAsync(&n_steps, steps + n_slices, 4, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  CUDA_TRY(b->plan_mem.alloc(
      {GROUP_PART(b->pp_idx, (size_t)n_steps * S * kPprU * 4),
       GROUP_PART(b->pp_step_off, ((size_t)n_slices + 1) * 4),
       GROUP_PART(b->pp_unit_dst, (size_t)n_slices * S * 4),
       GROUP_PART(b->pp_long_row, (size_t)total[2] * 4),
       GROUP_PART(b->pp_long_slot, ((size_t)total[2] + 1) * 4)}));
  if (n_slices > 0)
    k_plan_index<<<grid, kNT, 0, s>>>(place, steps, e->csc_src, U, S, n_slices, e->nV, b->pp_idx,
                                     unit_dst);
  CUDA_TRY(cudaGetLastError());
  const struct {
    int32_t *to, *from;
    size_t n;
  } keep[] = {{b->pp_step_off, steps, (size_t)n_slices + 1},
              {b->pp_unit_dst, unit_dst, (size_t)n_slices * S},
              {b->pp_long_row, long_row, (size_t)total[2]},
              {b->pp_long_slot, long_slot, (size_t)total[2] + 1}};
  for (const auto &k : keep)
    if (k.n) CUDA_TRY(cudaMemcpyAsync(k.to, k.from, k.n * 4, cudaMemcpyDeviceToDevice, s));
  CUDA_TRY(cudaStreamSynchronize(s));  // the scratch is freed at return
  b->n_slices = n_slices;
  b->n_steps = n_steps;
  b->n_slots = total[1];
  b->n_long = total[2];
  b->plan_S = S;
  return GAS_OK;
}

// Ranks, contributions and row sums of the lanes; the gather's plan for their
// groups and its pieces of P edges per group.
gas_status_t ensure_ppr(gas_batch *b, int lanes, int P, int n_seeds, int grid_rows,
                        cudaStream_t s) {
  gas_engine *e = b->eng;
  const size_t nV = std::max(1, e->nV), n_ne = std::max(1, e->n_ne);
  const int G = lane_group(lanes), S = 32 / (G / ppr_vl(lanes));
  if (b->plan_S != S) {
    drop_graph(b);
    b->ppr_lanes = 0;  // the partials are sized by the plan
    GAS_TRY(build_ppr_plan(b, S, s));
  }
  if (b->ppr_lanes != lanes) {
    drop_graph(b);
    b->ppr_lanes = 0;
    const size_t row = (size_t)lanes * 4;
    CUDA_TRY(b->ppr_mem.alloc({GROUP_PART(b->rank, nV * row),
                               GROUP_PART(b->contrib, (nV + 1) * row),
                               GROUP_PART(b->sum, n_ne * row),
                               GROUP_PART(b->partial, (size_t)b->n_slots * lanes * sizeof(CVal))}));
    b->ppr_lanes = lanes;
    b->piece_edges = 0;
  }
  if (!b->seed_mask) CUDA_TRY(renew(b->seed_mask, nV * 4));
  if (!b->ticket) {
    CUDA_TRY(renew(b->ticket, 4));
    CUDA_TRY(cudaMemsetAsync(b->ticket, 0, 4, s));
  }
  if (b->seeds_cap < n_seeds) {
    drop_graph(b);
    b->seeds_cap = 0;
    CUDA_TRY(renew(b->seeds, (size_t)n_seeds * 4));
    b->seeds_cap = n_seeds;
  }
  const int need_l1 = grid_rows * G;
  if (b->l1_cap < need_l1) {
    drop_graph(b);
    b->l1_cap = 0;
    CUDA_TRY(renew(b->l1, (size_t)need_l1 * sizeof(double)));
    b->l1_cap = need_l1;
  }
  if (b->piece_edges == P) return GAS_OK;
  drop_graph(b);
  b->piece_edges = 0;
  const int steps = (P + kPprU - 1) / kPprU;
  const int n_pieces = (int)(((long long)b->n_steps + steps - 1) / steps);
  CUDA_TRY(b->piece_mem.alloc({GROUP_PART(b->pp_piece_start, ((size_t)n_pieces + 1) * 4)}));
  k_plan_pieces<<<8 * e->num_sms, 256, 0, s>>>(b->pp_step_off, b->n_slices, n_pieces, steps,
                                              b->pp_piece_start);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaStreamSynchronize(s));  // the plan outlives this call and its stream
  b->n_pieces = n_pieces;
  b->piece_edges = P;
  return GAS_OK;
}

struct RunCtx {
  gas_batch *b;
  int bfs_lanes, ppr_lanes, sssp_lanes;
  int slab_grid, grid_pieces, grid_fix, grid_rows, sssp_grid;
  PprArgs ppr;
};

PprArgs ppr_args(gas_batch *b, int lanes) {
  gas_engine *e = b->eng;
  PprArgs a;
  a.csc_off = e->csc_off;
  a.csr_off = e->csr_off;
  a.ne_vid = e->ne_vid;
  a.idx = b->pp_idx;
  a.step_off = b->pp_step_off;
  a.unit_dst = b->pp_unit_dst;
  a.piece_start = b->pp_piece_start;
  a.long_row = b->pp_long_row;
  a.long_slot = b->pp_long_slot;
  a.n_pieces = b->n_pieces;
  a.n_long = b->n_long;
  a.L = lanes;
  a.G = lane_group(lanes);
  a.n_ne = e->n_ne;
  a.nV = e->nV;
  a.partial = b->partial;
  a.sum = b->sum;
  a.rank = b->rank;
  a.contrib = b->contrib;
  a.l1_part = b->l1;
  a.lane_resid = b->resid;
  a.ticket = b->ticket;
  a.seed_mask = b->seed_mask;
  a.prm = b->prm;
  a.cnt = b->cnt + 1;
  return a;
}

typedef gas_status_t (*StepFn)(RunCtx *, cudaStream_t, cudaGraphConditionalHandle, int);

// The next frontier of new lanes, then the loop control (first: the
// prologue's sources, level 0).
template <int WW>
gas_status_t bfs_compact_w(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig,
                           int first) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  const int nb = ms_blocks(b);
  const int L = c->bfs_lanes, ng = (int)b->v_off.size() - 1;
  k_ms_count<WW><<<nb, kNT, 0, s>>>(b->tbits, nullptr, b->vn, e->csr_off, nwords(b), b->qpart,
                                ms_wpart(b), nullptr, b->dir);
  k_mss_spine<<<1, kMssSpineNT, 0, s>>>(reinterpret_cast<int2 *>(b->qpart), nb, b->cnt,
                                        c->slab_grid * (kNT / 32), b->edges, nullptr, nullptr,
                                        b->dir, b->alive, ng, (unsigned long long)e->nE * L,
                                        e->nV, h, ig, first);
  k_ms_write<WW><<<nb, kNT, 0, s>>>(b->tbits, b->vn, e->csr_off, nwords(b), b->qpart,
                               ms_wpart(b), L, lane_group(L), b->cnt, b->depth, b->q_mask,
                               b->q_end, b->q_delta, b->part, b->fr, b->alive, b->g_off, ng,
                               e->nV);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

gas_status_t bfs_compact(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig,
                         int first) {
  switch (ms_words(c->b)) {
    case 2: return bfs_compact_w<2>(c, s, h, ig, first);
    case 4: return bfs_compact_w<4>(c, s, h, ig, first);
    default: return bfs_compact_w<16>(c, s, h, ig, first);
  }
}

gas_status_t bfs_prologue(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  const size_t nV = std::max(1, e->nV), nW = std::max(1, nwords(b));
  const int L = c->bfs_lanes;
  k_b_reset<<<1, 1, 0, s>>>(b->cnt, b->prm, 0, b->edges);
  CUDA_TRY(cudaMemsetAsync(b->vn, 0, nV * 8, s));
  CUDA_TRY(cudaMemsetAsync(b->tbits, 0, nW * 4, s));
  CUDA_TRY(cudaMemsetAsync(b->depth, 0xff, nV * L * 4, s));
  k_ms_seed<<<2 * e->num_sms, 256, 0, s>>>(b->srcs, b->prm, L, b->vn, b->tbits);
  return bfs_compact(c, s, h, ig, 1);
}

gas_status_t bfs_push(RunCtx *c, cudaStream_t s) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  const gasdev::SlabSource q = gasdev::slab_source(
      b->q_end, nullptr, b->q_delta, 0, 0, &b->cnt->n_changed, &b->cnt->n_scatter_edges,
      b->part, &b->cnt->push_chunk_log2);
  MsPushPol pol{e->csr_dst, b->q_mask, b->vn, b->tbits};
  const MsPull pull{e->csc_off, e->csc_src, b->fr, b->alive, b->g_off,
                    (int)b->v_off.size() - 1, e->nV};
  k_ms_level<<<c->slab_grid, kNT, 0, s>>>(pol, q, pull, b->cnt);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

gas_status_t bfs_body(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  gas_batch *b = c->b;
  if (b->profiling && !ig) {  // direct launches: the counters were just read
    // algorithmic bytes: per union edge its index and the destination's
    // visited and next words; per queue entry its edge range and lane mask
    const gas_counters &k = b->h_cnt[0];
    CUDA_TRY(cudaEventRecord(b->pev[0], s));
    GAS_TRY(bfs_push(c, s));
    CUDA_TRY(cudaEventRecord(b->pev[1], s));
    CUDA_TRY(cudaEventSynchronize(b->pev[1]));
    float ms = 0.f;
    CUDA_TRY(cudaEventElapsedTime(&ms, b->pev[0], b->pev[1]));
    if (k.mode == kModePull) {  // the dense reads only: visited, next, offsets
      b->prof.pull_ms += ms;
      b->prof.pull_bytes += 12LL * b->eng->nV;
      b->prof.pull_launches += 1;
    } else {
      b->prof.push_ms += ms;
      b->prof.push_bytes += (int64_t)k.n_scatter_edges * 12 + (int64_t)k.n_changed * 12;
      b->prof.push_launches += 1;
    }
  } else {
    GAS_TRY(bfs_push(c, s));
  }
  return bfs_compact(c, s, h, ig, 0);
}

// The queue of the changed lanes, then the loop control (first: the
// prologue's queue).
template <int WW>
gas_status_t sssp_compact_w(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig,
                            int first) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  const int nb = ms_blocks(b);
  k_ms_count<WW><<<nb, kNT, 0, s>>>(b->tbits, b->next, nullptr, e->csr_off, nwords(b), b->qpart,
                                ms_wpart(b), b->lanes_active, nullptr);
  k_mss_spine<<<1, kMssSpineNT, 0, s>>>(reinterpret_cast<int2 *>(b->qpart), nb, b->cnt + 2,
                                        c->sssp_grid * (kNT / 32), b->sssp_edges,
                                        b->lanes_active, b->lane_rounds, nullptr, nullptr, 0,
                                        0ull, 0, h, ig, first);
  k_mss_write<WW><<<nb, kNT, 0, s>>>(b->tbits, b->next, e->csr_off, nwords(b), b->qpart,
                                 ms_wpart(b), b->dist_ls, b->dist, b->q_mask, b->q_vals, b->q_end,
                                 b->q_delta, b->part, b->cnt + 2);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

gas_status_t sssp_compact(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig,
                          int first) {
  switch (ms_words(c->b)) {
    case 2: return sssp_compact_w<2>(c, s, h, ig, first);
    case 4: return sssp_compact_w<4>(c, s, h, ig, first);
    default: return sssp_compact_w<16>(c, s, h, ig, first);
  }
}

gas_status_t sssp_prologue(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  const size_t nV = std::max(1, e->nV), nW = std::max(1, nwords(b));
  k_b_reset<<<1, 1, 0, s>>>(b->cnt + 2, b->prm, 2, b->sssp_edges);
  CUDA_TRY(cudaMemsetAsync(b->next, 0, nV * 4, s));
  CUDA_TRY(cudaMemsetAsync(b->tbits, 0, nW * 4, s));
  k_mss_init<<<8 * e->num_sms, 256, 0, s>>>(b->dist, nV * b->dist_ls, b->lanes_active,
                                           b->lane_rounds);
  k_mss_seed<<<2 * e->num_sms, 256, 0, s>>>(b->sssp_srcs, b->prm, c->sssp_lanes, b->dist_ls,
                                           b->dist, b->next, b->tbits);
  return sssp_compact(c, s, h, ig, 1);
}

gas_status_t sssp_push(RunCtx *c, cudaStream_t s) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  const gasdev::SlabSource q = gasdev::slab_source(
      b->q_end, nullptr, b->q_delta, 0, 0, &b->cnt[2].n_changed, &b->cnt[2].n_scatter_edges,
      b->part, &b->cnt[2].push_chunk_log2);
  const int32_t *w = b->weighted ? (const int32_t *)e->csr_ed : nullptr;
  if (b->dist_ls == 4) {
    MssPushPolStaged<1> pol{e->csr_dst, w, b->q_vals, b->dist, b->next, b->tbits};
    k_mss_push<<<c->sssp_grid, kNT, 0, s>>>(pol, q);
  } else if (b->dist_ls == 8) {
    MssPushPolStaged<2> pol{e->csr_dst, w, b->q_vals, b->dist, b->next, b->tbits};
    k_mss_push<<<c->sssp_grid, kNT, 0, s>>>(pol, q);
  } else {
    MssPushPol pol{e->csr_dst, w, b->q_mask, b->q_vals, b->dist, b->next, b->tbits,
                   b->dist_ls};
    k_mss_push<<<c->sssp_grid, kNT, 0, s>>>(pol, q);
  }
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

// Algorithmic bytes of one SSSP push: per union edge its index, its weight
// and the destination row; per queue entry its edge range and snapshot row.
int64_t sssp_push_bytes(const gas_batch *b, const gas_counters &c) {
  const int64_t row = 4LL * b->dist_ls;
  return (int64_t)c.n_scatter_edges * ((b->weighted ? 8 : 4) + row) +
         (int64_t)c.n_changed * (8 + row);
}

gas_status_t sssp_body(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  gas_batch *b = c->b;
  if (b->profiling && !ig) {  // direct launches: the counters were just read
    CUDA_TRY(cudaEventRecord(b->pev[0], s));
    GAS_TRY(sssp_push(c, s));
    CUDA_TRY(cudaEventRecord(b->pev[1], s));
    CUDA_TRY(cudaEventSynchronize(b->pev[1]));
    float ms = 0.f;
    CUDA_TRY(cudaEventElapsedTime(&ms, b->pev[0], b->pev[1]));
    b->prof.push_ms += ms;
    b->prof.push_bytes += sssp_push_bytes(b, b->h_cnt[2]);
    b->prof.push_launches += 1;
  } else {
    GAS_TRY(sssp_push(c, s));
  }
  return sssp_compact(c, s, h, ig, 0);
}

gas_status_t ppr_prologue(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  gas_batch *b = c->b;
  gas_engine *e = b->eng;
  k_b_reset<<<1, 1, 0, s>>>(b->cnt + 1, b->prm, 1, nullptr);
  CUDA_TRY(cudaMemsetAsync(b->seed_mask, 0, (size_t)std::max(1, e->nV) * 4, s));
  k_ppr_seed<<<2 * e->num_sms, 256, 0, s>>>(b->seeds, b->prm, c->ppr_lanes, b->seed_mask);
  k_ppr_init<<<8 * e->num_sms, 256, 0, s>>>(b->seed_mask, e->csr_off, e->nV, c->ppr_lanes,
                                           b->rank, b->contrib);
  k_ppr_precond<<<1, 1, 0, s>>>(b->cnt + 1, h, ig);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

template <int VL>
gas_status_t ppr_step(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  k_ppr_units<VL><<<c->grid_pieces, kNT, 0, s>>>(c->ppr);
  k_ppr_fix<VL><<<c->grid_fix, kNT, 0, s>>>(c->ppr);
  k_ppr_rows<VL><<<c->grid_rows, kNT, 0, s>>>(c->ppr, h, ig);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

gas_status_t ppr_body(RunCtx *c, cudaStream_t s, cudaGraphConditionalHandle h, int ig) {
  switch (ppr_vl(c->ppr_lanes)) {
    case 4: return ppr_step<4>(c, s, h, ig);
    case 2: return ppr_step<2>(c, s, h, ig);
    default: return ppr_step<1>(c, s, h, ig);
  }
}

struct Loop {
  StepFn pro, body;
};

// One graph: for each loop, its prologue then WHILE(cond) { body }.
gas_status_t build_chain(RunCtx *c, const Loop *loops, int n, cudaGraphExec_t *out) {
  cudaGraph_t g = nullptr;
  cudaStream_t cs = nullptr;
  gas_status_t st = GAS_OK;
  CUDA_TRY(cudaGraphCreate(&g, 0));
  cudaError_t ce = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (ce != cudaSuccess) {
    cudaGraphDestroy(g);
    return fail(GAS_ERR_CUDA, "batch graph stream: %s", cudaGetErrorString(ce));
  }
  cudaGraphNode_t prev = nullptr;
  for (int i = 0; i < n && st == GAS_OK; ++i) {
    cudaGraphConditionalHandle h;
    ce = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
    if (ce == cudaSuccess)
      ce = cudaStreamBeginCaptureToGraph(cs, g, prev ? &prev : nullptr, nullptr, prev ? 1 : 0,
                                         cudaStreamCaptureModeRelaxed);
    if (ce != cudaSuccess) {
      st = fail(GAS_ERR_CUDA, "batch prologue capture: %s", cudaGetErrorString(ce));
      break;
    }
    st = loops[i].pro(c, cs, h, 1);
    std::vector<cudaGraphNode_t> deps;
    if (st == GAS_OK) {
      cudaStreamCaptureStatus cst;
      const cudaGraphNode_t *d = nullptr;
      size_t nd = 0;
      ce = cudaStreamGetCaptureInfo(cs, &cst, nullptr, nullptr, &d, nullptr, &nd);
      if (ce == cudaSuccess) deps.assign(d, d + nd);
      else st = fail(GAS_ERR_CUDA, "capture info: %s", cudaGetErrorString(ce));
    }
    cudaGraph_t cap = nullptr;
    ce = cudaStreamEndCapture(cs, &cap);
    if (st == GAS_OK && ce != cudaSuccess)
      st = fail(GAS_ERR_CUDA, "end prologue capture: %s", cudaGetErrorString(ce));
    if (st != GAS_OK) break;
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    ce = cudaGraphAddNode(&node, g, deps.data(), nullptr, deps.size(), &p);
    if (ce != cudaSuccess) {
      st = fail(GAS_ERR_CUDA, "add while node: %s", cudaGetErrorString(ce));
      break;
    }
    ce = cudaStreamBeginCaptureToGraph(cs, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                       cudaStreamCaptureModeRelaxed);
    if (ce != cudaSuccess) {
      st = fail(GAS_ERR_CUDA, "body capture: %s", cudaGetErrorString(ce));
      break;
    }
    st = loops[i].body(c, cs, h, 1);
    cudaGraph_t bc = nullptr;
    ce = cudaStreamEndCapture(cs, &bc);
    if (st == GAS_OK && ce != cudaSuccess)
      st = fail(GAS_ERR_CUDA, "end body capture: %s", cudaGetErrorString(ce));
    prev = node;
  }
  if (st == GAS_OK) {
    ce = cudaGraphInstantiate(out, g, 0);
    if (ce != cudaSuccess) st = fail(GAS_ERR_CUDA, "instantiate: %s", cudaGetErrorString(ce));
  }
  cudaStreamDestroy(cs);
  cudaGraphDestroy(g);
  return st;
}

// The same loops as direct launches with one host read of the condition per
// iteration (GAS_HOST_LOOP=1: ncu cannot profile kernels inside graphs with
// conditional nodes).
gas_status_t run_direct(RunCtx *c, const Loop *loops, const int *which, int n, cudaStream_t s) {
  gas_batch *b = c->b;
  for (int i = 0; i < n; ++i) {
    GAS_TRY(loops[i].pro(c, s, 0, 0));
    for (;;) {
      CUDA_TRY(cudaMemcpyAsync(b->h_cnt + which[i], b->cnt + which[i], sizeof(gas_counters),
                               cudaMemcpyDeviceToHost, s));
      CUDA_TRY(cudaStreamSynchronize(s));
      if (!b->h_cnt[which[i]].cond) break;
      GAS_TRY(loops[i].body(c, s, 0, 0));
    }
  }
  return GAS_OK;
}

// Resident CTAs of the PPR kernels.
template <int VL>
void ppr_grids(const gas_engine *e, RunCtx *c) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ppr_units<VL>, kNT, 0);
  c->grid_pieces = e->num_sms * (per_sm > 0 ? per_sm : 1);
  per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ppr_fix<VL>, kNT, 0);
  c->grid_fix = e->num_sms * (per_sm > 0 ? per_sm : 1);
  per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ppr_rows<VL>, kNT, 0);
  c->grid_rows = e->num_sms * (per_sm > 0 ? per_sm : 1);
}

void grids(gas_batch *b, RunCtx *c) {
  gas_engine *e = b->eng;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ms_level, kNT, 0);
  c->slab_grid = e->num_sms * (per_sm > 0 ? per_sm : 1);
  switch (ppr_vl(c->ppr_lanes)) {
    case 4: ppr_grids<4>(e, c); break;
    case 2: ppr_grids<2>(e, c); break;
    default: ppr_grids<1>(e, c); break;
  }
  per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mss_push<MssPushPolStaged<2>>, kNT,
                                                0);
  c->sssp_grid = e->num_sms * (per_sm > 0 ? per_sm : 1);
}

gas_status_t check_job(const gas_batch *b, const gas_batch_job *j) {
  if (!j) return fail(GAS_ERR_INVALID, "null job");
  if (j->bfs_lanes < 0 || j->bfs_lanes > kMaxLanes || j->ppr_lanes < 0 ||
      j->ppr_lanes > kMaxLanes || j->sssp_lanes < 0 || j->sssp_lanes > kMaxLanes)
    return fail(GAS_ERR_INVALID, "lanes must be in [0, %d]", kMaxLanes);
  if (j->bfs_lanes == 0 && j->ppr_lanes == 0 && j->sssp_lanes == 0)
    return fail(GAS_ERR_INVALID, "job has no BFS, SSSP or PPR lanes");
  if (j->bfs_lanes > 0 && !j->bfs_sources) return fail(GAS_ERR_INVALID, "null bfs_sources");
  if (j->sssp_lanes > 0 && !j->sssp_sources)
    return fail(GAS_ERR_INVALID, "null sssp_sources");
  if (j->ppr_lanes > 0) {
    if (!j->ppr_seeds) return fail(GAS_ERR_INVALID, "null ppr_seeds");
    if (!(j->damping > 0.0 && j->damping < 1.0) || !(j->tol > 0.0))
      return fail(GAS_ERR_INVALID, "damping must be in (0,1), tol > 0");
  }
  if (j->piece_edges < 0 || j->piece_edges > (1 << 20))
    return fail(GAS_ERR_INVALID, "piece_edges must be in [0, 2^20]");
  const int G = (int)b->v_off.size() - 1;
  for (int pass = 0; pass < 3; ++pass) {
    const int L = pass == 0 ? j->bfs_lanes : pass == 1 ? j->ppr_lanes : j->sssp_lanes;
    const int32_t *ids = pass == 0 ? j->bfs_sources : pass == 1 ? j->ppr_seeds : j->sssp_sources;
    for (int g = 0; g < G; ++g)
      for (int l = 0; l < L; ++l) {
        const int32_t s = ids[(size_t)g * L + l];
        if (s < -1 || s >= b->v_off[g + 1] - b->v_off[g])
          return fail(GAS_ERR_INVALID, "%s %d of graph %d lane %d out of range",
                      pass == 1 ? "seed" : "source", s, g, l);
      }
  }
  return GAS_OK;
}

// Untuned piece size: 256, halved down to 64 while there would be fewer than
// 1.5 pieces per resident group (16 lanes on 600 K edges: 64 takes 0.74 ms
// per run, 256 0.96; on 64 M edges 11.3 and 10.0).
int default_piece(const gas_batch *b, const RunCtx &c) {
  if (b->tuned_piece > 0) return b->tuned_piece;
  const int L = std::max(1, c.ppr_lanes);
  const int64_t groups = (int64_t)c.grid_pieces * (kNT / (lane_group(L) / ppr_vl(L)));
  int P = 256;
  while (P > 64 && (int64_t)b->eng->nE / P * 2 < groups * 3) P /= 2;
  return P;
}

}  // namespace

extern "C" {

gas_status_t gas_batch_create(gas_batch **out) {
  if (!out) return fail(GAS_ERR_INVALID, "null out");
  *out = nullptr;
  gas_batch *b = new (std::nothrow) gas_batch;
  if (!b) return fail(GAS_ERR_NOMEM, "batch");
  gas_status_t st = gas_engine_create(GAS_PROG_BFS, &b->eng);
  if (st != GAS_OK) {
    delete b;
    return st;
  }
  *out = b;
  return GAS_OK;
}

void gas_batch_destroy(gas_batch *b) {
  if (!b) return;
  free_state(b);
  for (cudaEvent_t &ev : b->pev)
    if (ev) cudaEventDestroy(ev);
  bfree(b->cnt);
  bfree(b->prm);
  bfree(b->edges);
  bfree(b->sssp_edges);
  bfree(b->resid);
  if (b->h_cnt) cudaFreeHost(b->h_cnt);
  gas_engine_destroy(b->eng);
  delete b;
}

gas_status_t gas_batch_add_graph(gas_batch *b, int32_t nV, int64_t nE, const int32_t *srcs,
                                 const int32_t *dsts, int32_t *graph_id) {
  return gas_batch_add_graph_weighted(b, nV, nE, srcs, dsts, nullptr, graph_id);
}

gas_status_t gas_batch_add_graph_weighted(gas_batch *b, int32_t nV, int64_t nE,
                                          const int32_t *srcs, const int32_t *dsts,
                                          const int32_t *weights, int32_t *graph_id) {
  if (!b || nV < 0 || nE < 0 || (nE > 0 && (!srcs || !dsts)))
    return fail(GAS_ERR_INVALID, "batch_add_graph: bad arguments");
  if (b->built) return fail(GAS_ERR_STATE, "batch already built");
  const int64_t base = b->v_off.back();
  if (base + nV > INT32_MAX - 1 || b->n_edges + nE > INT32_MAX - 1)
    return fail(GAS_ERR_TOO_LARGE, "batch exceeds the 32-bit index space");
  for (int64_t i = 0; i < nE; ++i)
    if (srcs[i] < 0 || srcs[i] >= nV || dsts[i] < 0 || dsts[i] >= nV)
      return fail(GAS_ERR_INVALID, "batch_add_graph: edge %lld outside [0, %d)",
                  (long long)i, nV);
  if (weights)  // the SSSP Program's margin: dist + w never passes INT_MAX
    for (int64_t i = 0; i < nE; ++i)
      if (weights[i] < 0 || weights[i] > 100000)
        return fail(GAS_ERR_INVALID, "batch_add_graph: weight %d of edge %lld outside "
                    "[0, 100000]", weights[i], (long long)i);
  try {
    const size_t n0 = b->src.size();
    b->src.resize(n0 + nE);
    b->dst.resize(n0 + nE);
    for (int64_t i = 0; i < nE; ++i) {
      b->src[n0 + i] = (int32_t)(srcs[i] + base);
      b->dst[n0 + i] = (int32_t)(dsts[i] + base);
    }
    if (weights && !b->weighted) {  // earlier graphs weigh 1 per edge
      b->w.assign(n0, 1);
      b->weighted = true;
    }
    if (b->weighted) {
      b->w.resize(n0 + nE, 1);
      if (weights) std::copy(weights, weights + nE, b->w.begin() + n0);
    }
    b->v_off.push_back((int32_t)(base + nV));
  } catch (...) {
    return fail(GAS_ERR_NOMEM, "batch edge list");
  }
  b->n_edges += nE;
  if (graph_id) *graph_id = (int32_t)b->v_off.size() - 2;
  return GAS_OK;
}

gas_status_t gas_batch_build(gas_batch *b, void *stream) {
  if (!b) return fail(GAS_ERR_INVALID, "null batch");
  if (b->built) return fail(GAS_ERR_STATE, "batch already built");
  if (b->v_off.size() < 2) return fail(GAS_ERR_STATE, "batch has no graphs");
  const int32_t nV = b->v_off.back();
  if (b->weighted) {  // an engine whose graph carries int32 edge data
    gas_engine *we = nullptr;
    GAS_TRY(gas_engine_create(GAS_PROG_SSSP, &we));
    gas_engine_destroy(b->eng);
    b->eng = we;
  }
  b->eng->graph_only = true;
  std::vector<int32_t> vd((size_t)std::max(1, nV), -1);
  GAS_TRY(gas_engine_set_graph(b->eng, nV, vd.data(), (int64_t)b->src.size(),
                               b->weighted ? b->w.data() : nullptr, b->src.data(),
                               b->dst.data(), stream));
  if (!b->cnt) {
    CUDA_TRY(cudaMalloc(&b->cnt, 3 * sizeof(gas_counters)));
    CUDA_TRY(cudaMemsetAsync(b->cnt, 0, 3 * sizeof(gas_counters), (cudaStream_t)stream));
    CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));  // runs take other streams
    CUDA_TRY(cudaMallocHost(&b->h_cnt, 3 * sizeof(gas_counters)));
    CUDA_TRY(cudaMalloc(&b->prm, sizeof(BatchParams)));
    CUDA_TRY(cudaMalloc(&b->edges, sizeof(unsigned long long)));
    CUDA_TRY(cudaMalloc(&b->sssp_edges, sizeof(unsigned long long)));
    CUDA_TRY(cudaMalloc(&b->resid, (1 + kMaxLanes) * sizeof(double)));
  }
  std::vector<int32_t>().swap(b->src);
  std::vector<int32_t>().swap(b->dst);
  std::vector<int32_t>().swap(b->w);
  // the traversals' frontier (four words per vertex, and a word per 64 edges),
  // so that the first run finds it; that run asks again where it is more than
  // a quarter of the free memory, as a batch may only ever run PPR
  if (gas::within_quarter_of_free((size_t)nV * 17 + (size_t)b->n_edges / 16) &&
      ensure_frontier(b) != GAS_OK)
    gas::clear_error();
  b->built = true;
  return GAS_OK;
}

int32_t gas_batch_num_graphs(const gas_batch *b) {
  return b ? (int32_t)b->v_off.size() - 1 : 0;
}

int32_t gas_batch_num_vertices(const gas_batch *b) { return b ? b->v_off.back() : 0; }

int64_t gas_batch_num_edges(const gas_batch *b) { return b ? b->n_edges : 0; }

int32_t gas_batch_vertex_offset(const gas_batch *b, int32_t g) {
  return (b && g >= 0 && g < (int32_t)b->v_off.size()) ? b->v_off[g] : -1;
}

gas_status_t gas_batch_run(gas_batch *b, const gas_batch_job *job, int32_t *depth_out,
                           int32_t *dist_out, float *rank_out, gas_batch_stats *stats,
                           void *stream) {
  if (!b || !b->built) return fail(GAS_ERR_STATE, "batch not built");
  GAS_TRY(check_job(b, job));
  gas_engine *e = b->eng;
  cudaStream_t s = S(stream);
  const int G = gas_batch_num_graphs(b), nV = e->nV;
  const int LB = job->bfs_lanes, LP = job->ppr_lanes, LS = job->sssp_lanes;
  if (stats) *stats = gas_batch_stats{};
  RunCtx c;
  c.b = b;
  c.bfs_lanes = LB;
  c.ppr_lanes = LP;
  c.sssp_lanes = LS;
  grids(b, &c);
  const int P = job->piece_edges > 0 ? job->piece_edges : default_piece(b, c);
  BatchParams prm{};
  prm.damping = LP ? job->damping : 0.85;
  prm.tol = LP ? job->tol : 1.0;
  prm.bfs_max_iter = job->max_bfs_levels > 0 ? job->max_bfs_levels : nV + 2;
  prm.ppr_max_iter = job->max_ppr_iterations > 0 ? job->max_ppr_iterations : 1000;
  prm.n_sources = G * LB;
  prm.sssp_max_iter = job->max_sssp_iterations > 0 ? job->max_sssp_iterations : nV + 2;
  prm.n_sssp_sources = G * LS;
  prm.n_seeds = G * LP;
  std::vector<int32_t> sg, ss;
  if (LB) {
    GAS_TRY(ensure_bfs(b, LB, G * LB, s));
    sg.resize((size_t)G * LB);
    for (int g = 0; g < G; ++g)
      for (int l = 0; l < LB; ++l) {
        const int32_t v = job->bfs_sources[(size_t)g * LB + l];
        sg[(size_t)g * LB + l] = v < 0 ? -1 : v + b->v_off[g];
      }
  }
  if (LS) {
    GAS_TRY(ensure_sssp(b, LS, G * LS));
    ss.resize((size_t)G * LS);
    for (int g = 0; g < G; ++g)
      for (int l = 0; l < LS; ++l) {
        const int32_t v = job->sssp_sources[(size_t)g * LS + l];
        ss[(size_t)g * LS + l] = v < 0 ? -1 : v + b->v_off[g];
      }
  }
  std::vector<int32_t> pg;
  if (LP) {
    gas_status_t st = ensure_ppr(b, LP, P, G * LP, c.grid_rows, s);
    if (st != GAS_OK && !LB && !LS && b->next) {
      // the traversals' frontier, which this run does not use, may have the
      // memory that it needs
      drop_graph(b);
      b->frontier_mem.free();
      gas::clear_error();
      st = ensure_ppr(b, LP, P, G * LP, c.grid_rows, s);
    }
    GAS_TRY(st);
    pg.resize((size_t)G * LP);
    for (int g = 0; g < G; ++g)
      for (int l = 0; l < LP; ++l) {
        const int32_t v = job->ppr_seeds[(size_t)g * LP + l];
        pg[(size_t)g * LP + l] = v < 0 ? -1 : v + b->v_off[g];
      }
    c.ppr = ppr_args(b, LP);
  }
  Loop loops[3];
  int which[3];
  int n = 0;
  if (LB) { loops[n] = Loop{bfs_prologue, bfs_body}; which[n++] = 0; }
  if (LS) { loops[n] = Loop{sssp_prologue, sssp_body}; which[n++] = 2; }
  if (LP) { loops[n] = Loop{ppr_prologue, ppr_body}; which[n++] = 1; }
  const bool direct = gas::host_loop_requested() || b->profiling;
  if (!direct && (!b->graph || b->g_bfs_lanes != LB || b->g_ppr_lanes != LP ||
                  b->g_sssp_lanes != LS || b->g_piece != (LP ? P : -1))) {
    drop_graph(b);
    GAS_TRY(build_chain(&c, loops, n, &b->graph));
    b->g_bfs_lanes = LB;
    b->g_ppr_lanes = LP;
    b->g_sssp_lanes = LS;
    b->g_piece = LP ? P : -1;
  }
  CUDA_TRY(cudaMemcpyAsync(b->prm, &prm, sizeof(prm), cudaMemcpyHostToDevice, s));
  if (LB) CUDA_TRY(cudaMemcpyAsync(b->srcs, sg.data(), sg.size() * 4, cudaMemcpyHostToDevice, s));
  if (LS)
    CUDA_TRY(cudaMemcpyAsync(b->sssp_srcs, ss.data(), ss.size() * 4, cudaMemcpyHostToDevice, s));
  if (LP)
    CUDA_TRY(cudaMemcpyAsync(b->seeds, pg.data(), pg.size() * 4, cudaMemcpyHostToDevice, s));
  if (direct) {
    GAS_TRY(run_direct(&c, loops, which, n, s));
  } else {
    CUDA_TRY(cudaGraphLaunch(b->graph, s));
  }
  CUDA_TRY(cudaMemcpyAsync(b->h_cnt, b->cnt, 3 * sizeof(gas_counters), cudaMemcpyDeviceToHost, s));
  unsigned long long edges = 0, sedges = 0;
  double resid[1 + kMaxLanes] = {};
  int32_t rounds[kMaxLanes] = {};
  if (LB) CUDA_TRY(cudaMemcpyAsync(&edges, b->edges, sizeof(edges), cudaMemcpyDeviceToHost, s));
  if (LS) {
    CUDA_TRY(cudaMemcpyAsync(&sedges, b->sssp_edges, sizeof(sedges), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaMemcpyAsync(rounds, b->lane_rounds, sizeof(rounds), cudaMemcpyDeviceToHost, s));
  }
  if (LP) CUDA_TRY(cudaMemcpyAsync(resid, b->resid, sizeof(resid), cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  const gas_counters cb = b->h_cnt[0], cp = b->h_cnt[1], cs = b->h_cnt[2];
  if (depth_out && LB)
    CUDA_TRY(cudaMemcpyAsync(depth_out, b->depth, (size_t)nV * LB * 4, cudaMemcpyDefault, s));
  if (dist_out && LS && nV > 0)  // rows of LS lanes in the device layout
    CUDA_TRY(cudaMemcpy2DAsync(dist_out, (size_t)LS * 4, b->dist, (size_t)b->dist_ls * 4,
                               (size_t)LS * 4, (size_t)nV, cudaMemcpyDefault, s));
  if (rank_out && LP)
    CUDA_TRY(cudaMemcpyAsync(rank_out, b->rank, (size_t)nV * LP * 4,
                             cudaMemcpyDefault, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (stats) {
    stats->bfs_iterations = LB ? cb.iteration : 0;
    stats->bfs_edges = (int64_t)edges;
    stats->ppr_iterations = LP ? cp.iteration : 0;
    stats->ppr_residual = resid[0];
    stats->piece_edges = LP ? P : 0;
    stats->sssp_iterations = LS ? cs.iteration : 0;
    stats->sssp_edges = (int64_t)sedges;
    for (int l = 0; l < LS; ++l) stats->sssp_lane_iterations[l] = rounds[l];
    // BFS: prologue 5 kernels (reset, seed, 3 compaction), 4 per level;
    // SSSP: prologue 6 (reset, init, seed, 3 compaction), 4 per iteration;
    // PPR: prologue 4 (reset, seeds, init, condition), 3 per iteration
    stats->kernel_launches = (LB ? 5 + 4 * cb.iteration : 0) +
                             (LS ? 6 + 4 * cs.iteration : 0) + (LP ? 4 + 3 * cp.iteration : 0);
    stats->graph_launches = direct ? 0 : 1;
    for (int l = 0; l < LP; ++l) stats->ppr_lane_residual[l] = resid[1 + l];
  }
  if (LS && cs.error) {
    CUDA_TRY(cudaMemsetAsync(&b->cnt[2].error, 0, sizeof(int32_t), s));
    CUDA_TRY(cudaStreamSynchronize(s));
    return fail(cs.error == GAS_ERR_ITER_CAP ? GAS_ERR_ITER_CAP : GAS_ERR_DEVICE,
                "batch sssp: device error %d after %d iterations", cs.error, cs.iteration);
  }
  if (LB && cb.error) {
    CUDA_TRY(cudaMemsetAsync(&b->cnt[0].error, 0, sizeof(int32_t), s));
    CUDA_TRY(cudaStreamSynchronize(s));
    return fail(cb.error == GAS_ERR_ITER_CAP ? GAS_ERR_ITER_CAP : GAS_ERR_DEVICE,
                "batch bfs: device error %d after %d levels", cb.error, cb.iteration);
  }
  if (LP && cp.error) {
    CUDA_TRY(cudaMemsetAsync(&b->cnt[1].error, 0, sizeof(int32_t), s));
    CUDA_TRY(cudaStreamSynchronize(s));
    return fail(cp.error == GAS_ERR_ITER_CAP ? GAS_ERR_ITER_CAP : GAS_ERR_DEVICE,
                "batch ppr: residual %.3e after %d iterations", resid[0], cp.iteration);
  }
  return GAS_OK;
}

gas_status_t gas_batch_set_profiling(gas_batch *b, int32_t on) {
  if (!b) return fail(GAS_ERR_INVALID, "null batch");
  if (on && !b->pev[0]) {
    CUDA_TRY(cudaEventCreate(&b->pev[0]));
    CUDA_TRY(cudaEventCreate(&b->pev[1]));
  }
  b->profiling = on != 0;
  return GAS_OK;
}

gas_status_t gas_batch_get_profile(gas_batch *b, gas_kernel_profile *out, int32_t reset) {
  if (!b || !out) return fail(GAS_ERR_INVALID, "bad arguments");
  *out = b->prof;
  if (reset) b->prof = gas_kernel_profile{};
  return GAS_OK;
}

gas_status_t gas_batch_tune(gas_batch *b, int32_t ppr_lanes, double damping, int32_t trials,
                            int32_t *piece_edges_out, float *ms_per_iter_out, void *stream) {
  if (!b || !b->built) return fail(GAS_ERR_STATE, "batch not built");
  if (ppr_lanes < 1 || ppr_lanes > kMaxLanes || !(damping > 0.0 && damping < 1.0))
    return fail(GAS_ERR_INVALID, "batch_tune: bad arguments");
  if (trials <= 0) trials = 3;
  gas_engine *e = b->eng;
  cudaStream_t s = S(stream);
  RunCtx c;
  c.b = b;
  c.bfs_lanes = 0;
  c.sssp_lanes = 0;
  c.ppr_lanes = ppr_lanes;
  grids(b, &c);
  BatchParams prm{};
  prm.damping = damping;
  prm.tol = 0.0;
  prm.ppr_max_iter = INT_MAX;
  prm.n_seeds = 1;
  CUDA_TRY(cudaMemcpyAsync(b->prm, &prm, sizeof(prm), cudaMemcpyHostToDevice, s));
  const int cands[] = {64, 128, 256, 512, 1024, 2048};
  int best = 0;
  float best_ms = 0.f;
  cudaEvent_t ev[2];
  CUDA_TRY(cudaEventCreate(&ev[0]));
  CUDA_TRY(cudaEventCreate(&ev[1]));
  gas_status_t st = GAS_OK;
  for (int P : cands) {
    st = ensure_ppr(b, ppr_lanes, P, 1, c.grid_rows, s);
    if (st != GAS_OK) break;
    c.ppr = ppr_args(b, ppr_lanes);
    // a seed in lane 0 of vertex 0 makes the timed iterations do real work
    const int32_t zero = 0;
    if (cudaMemcpyAsync(b->seeds, &zero, 4, cudaMemcpyHostToDevice, s) != cudaSuccess) {
      st = fail(GAS_ERR_CUDA, "batch_tune: seed upload");
      break;
    }
    st = ppr_prologue(&c, s, 0, 0);
    if (st == GAS_OK) st = ppr_body(&c, s, 0, 0);  // warm-up
    if (st != GAS_OK) break;
    cudaEventRecord(ev[0], s);
    for (int t = 0; t < trials && st == GAS_OK; ++t) st = ppr_body(&c, s, 0, 0);
    cudaEventRecord(ev[1], s);
    if (cudaEventSynchronize(ev[1]) != cudaSuccess) {
      st = fail(GAS_ERR_CUDA, "batch_tune: %s", cudaGetErrorString(cudaGetLastError()));
      break;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev[0], ev[1]);
    ms /= (float)trials;
    if (!best || ms < best_ms) {
      best = P;
      best_ms = ms;
    }
  }
  cudaEventDestroy(ev[0]);
  cudaEventDestroy(ev[1]);
  if (st != GAS_OK) return st;
  b->tuned_piece = best;
  drop_graph(b);
  if (piece_edges_out) *piece_edges_out = best;
  if (ms_per_iter_out) *ms_per_iter_out = best_ms;
  return GAS_OK;
}

}  // extern "C"
