// gas_small.cu -- BFS on graphs of up to 2^23 vertices as one persistent
// kernel.
//
// A BFS level is a few microseconds to some tens of them, and the fast
// schedule's per-level cost -- a WHILE iteration of the loop graph and its
// five kernel nodes, a pass that compacts the frontier -- is most of the run.
// Here one cooperative launch (every CTA resident) runs all levels:
// the same level sets as run() (the reference's pull-over-active loop,
// refgas.h:143-214 with bfs.cu:58-71's apply), top-down or bottom-up per
// level by the fast schedule's direction rule (PULL forces bottom-up, and
// PUSH keeps the fast schedule), with one grid barrier per level.
//
//   level 0      apply over the caller's active set: unvisited vertices get
//                depth 0 and form C_0;
//   top-down     the queue's entries (gas_stage.cuh) are spread over all
//                warps, each walking its entries' edges laid end to end, four
//                rounds of 32 in flight.  An unvisited target is claimed with
//                atomicCAS (-1 -> level), so exactly one thread adds it to
//                the next queue and sets its bit;
//   bottom-up    a thread per unvisited vertex scans its in-edges for a member
//                of C_k, the first alone and then four at a time (independent
//                loads), and stops at the first found; a row unfinished after
//                29 in-edges is taken over by its warp.  The warp writes whole
//                words of the next bitmap.
//
// A top-down level after a bottom-up or a big one first makes the queue from
// the bitmap, with a barrier of its own.  Iteration k+1 exists iff C_k has an
// out-edge (A_{k+1} = N(C_k)), so the count equals run()'s.  Frontier bitmaps
// rotate in three buffers (a level reads one, fills the next and clears the
// third).  Depths and bitmaps written by other SMs are read with plain loads:
// the barrier's acquire drops the SM's L1, and a depth read stale within a
// level (-1) only repeats a claim that fails.  The barrier's wait is bounded:
// past the limit every CTA leaves the kernel with an error.
//
// Bound by latency at every size: on R-MAT 65 K the warps wait at barriers (45
// cycles an issue; a level's chain is 5 to 10 us), on R-MAT 4 M for loads (12)
// and at barriers (11), with L1 at 17 % and L2 at 11 % of their peaks.
// Measured, us per run (before / here; before: one kernel with a warp per
// bitmap word and two barriers a top-down level up to 2^18 vertices, the
// multi-kernel loop above): R-MAT, 8 edges per vertex, 1 K 90 / 65, 16 K 108 /
// 69, 65 K 128 / 79, 250 K 178 / 89, 600 K 175 / 98, 1 M 203 / 104, 16 per
// vertex 4 M 317 / 194; Erdos-Renyi 100 K 138 / 83, 600 K 242 / 113, 2 M 257 /
// 160.  Above the old line over three or four graphs each, multi-kernel / here:
// R-MAT 4 M 283-335 / 186-200, directed 280-300 / 186-210, 8 M 421-455 /
// 313-360; Erdos-Renyi 4 M 424-473 / 252-271, 8 M 605-919 / 471-618.  Past the
// line, at 2^24: R-MAT 692-814 / 492-692, Erdos-Renyi 8 edges per vertex
// 1364-1448 / 1010-1059, but 16 per vertex 1040-1056 / 1242-1391.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "gas.h"
#include "gas_engine_impl.h"
#include "gas_internal.h"
#include "gas_sched.h"
#include "gas_stage.cuh"

namespace {

using namespace gasstage;

constexpr int kSbNT = kNT;          // one CTA per SM
constexpr int kSbAlone = 29;        // in-edges a thread looks at alone
// The direction rule of Beamer, Asanovic & Patterson (SC'12): bottom-up once
// the frontier's out-edges exceed 1/alpha of the edges not yet explored, then
// on while the frontier grows or holds more than V/beta vertices.
constexpr int kSbAlpha = 14;
constexpr int kSbBeta = 24;
constexpr int kSbCluster = 128;     // CTAs asked for up to which a cluster is enough (R-MAT
                                    // 16 K, 110 CTAs: 60 us against 68; 65 K, 450: 82 and 82)
constexpr int kSbDense = 2;         // out-edges per thread of the grid from which a
                                    // top-down level's finds are not queued (1 to 4
                                    // within 2 % of one another)

using gasgrid::warp_add;

struct SmallCtl {
  gasgrid::Barrier bar;
  Count q[3];       // of the level being read, filled and cleared (rotating)
  Count made[2];    // of queues made from a bitmap (in turn)
  long long bytes;  // algorithmic bytes (profiling)
};

struct Bfs {
  const int32_t *csr_off, *csr_dst, *csc_off, *csc_src;
  int32_t *depth;
  int nV;
};

// Top-down: the warp's share of a queue's light or heavy entries.  kBits: a
// big level -- its vertices are only marked and counted (edges, members),
// for a bottom-up level needs no queue and a top-down one makes it from the
// bitmap; appending 800 K vertices vertex by vertex took 200 us.
template <bool kCount, bool kBits>
__device__ __forceinline__ void sb_walk(const Bfs &g, const int4 *Q, int nq, int most, int w0,
                                        int level, uint32_t *N, int (*s_row)[3], Stage &st,
                                        const Queue &next, Count *ctr, int &edges, int &members,
                                        long long &bytes) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kRounds = 4;
  const int lane = threadIdx.x & 31;
  const int nwarps = gridDim.x * kWarps;
  int gwarp = dealt_warp() - w0;
  if (gwarp < 0) gwarp += nwarps;
  const int per = min(most, (nq + nwarps - 1) / nwarps);
  for (long long base = (long long)gwarp * per; base < nq; base += (long long)nwarps * per) {
    int start = 0, deg = 0;
    if (lane < per && base + lane < nq) {
      const int4 e = Q[base + lane];
      start = e.y;
      deg = e.z;
      if (kCount) bytes += 12 + 8LL * deg;
    }
    Rows rows;
    const int T = lay_out(start, deg, 0, s_row, rows);
    for (int r = 0; r < T; r += 32 * kRounds) {
      int v[kRounds];
      bool open[kRounds];
#pragma unroll
      for (int h = 0; h < kRounds; ++h) {
        const int r0 = r + 32 * h;
        const int pos = r0 + lane + __shfl_sync(FULL, rows.shift, row_of(rows, r0));
        v[h] = r0 + lane < T ? ld_edge(g.csr_dst + pos) : -1;
      }
#pragma unroll
      for (int h = 0; h < kRounds; ++h) open[h] = v[h] >= 0 && g.depth[v[h]] == -1;
#pragma unroll
      for (int h = 0; h < kRounds; ++h)
        if (!open[h] || atomicCAS(g.depth + v[h], -1, level) != -1) v[h] = -1;
#pragma unroll
      for (int h = 0; h < kRounds; ++h)
        if (v[h] >= 0) atomicOr(N + (v[h] >> 5), 1u << (v[h] & 31));
      if constexpr (kBits) {
#pragma unroll
        for (int h = 0; h < kRounds; ++h)
          if (v[h] >= 0) {
            edges += __ldg(g.csr_off + v[h] + 1) - __ldg(g.csr_off + v[h]);
            ++members;
          }
      } else {
        offer(st, v, g.csr_off, next, ctr);
      }
    }
  }
}

// Bottom-up: a warp per word of 32 vertices.  A word's chain is depth -> row
// offsets -> first in-edge -> frontier bit, so the loads of three words are
// in flight: the depths of the word two ahead, the offsets of the next one's
// unvisited rows, their first in-edges.  Adds the level's vertices and their
// out-edges to the thread's sums.
template <bool kCount>
__device__ __forceinline__ void sb_pull(const Bfs &g, const uint32_t *F, uint32_t *N, int nW,
                                        int level, int &edges, int &members, long long &bytes) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nwarps = gridDim.x * kWarps;
  auto depth_of = [&](long long w) {
    const long long v = (w << 5) + lane;
    return w < nW && v < g.nV ? g.depth[v] : 0;
  };
  int w = (blockIdx.x * kNT + threadIdx.x) >> 5;
  // word w: offsets and first in-edge; w + nwarps: offsets; w + 2 nwarps: depth
  int b0 = 0, e0 = 0, b1 = 0, e1 = 0, u0 = 0;
  {
    const bool in = depth_of(w) == -1;
    if (in) {
      b0 = __ldg(g.csc_off + (w << 5) + lane);
      e0 = __ldg(g.csc_off + (w << 5) + lane + 1);
    }
  }
  int d1 = depth_of((long long)w + nwarps);
  if (b0 < e0) u0 = __ldg(g.csc_src + b0);
  for (; w < nW; w += nwarps) {
    const int v = (w << 5) + lane;
    const int d2 = depth_of((long long)w + 2LL * nwarps);
    b1 = e1 = 0;
    if (d1 == -1) {
      b1 = __ldg(g.csc_off + v + 32 * nwarps);
      e1 = __ldg(g.csc_off + v + 32 * nwarps + 1);
    }
    uint32_t i = b0;  // unsigned: the steps past the last edge must not wrap
    const uint32_t end = e0;
    const uint32_t stop = end - i > kSbAlone ? i + kSbAlone : end;
    if (kCount) bytes += (v < g.nV ? 4 : 0) + (i < end ? 16 : 0);
    bool hit = i < end && ((F[u0 >> 5] >> (u0 & 31)) & 1u);
    for (++i; i < stop && !hit; i += 4) {
      int u[4];
      uint32_t f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = i + j < stop ? __ldg(g.csc_src + i + j) : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = u[j] >= 0 ? F[u[j] >> 5] : 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) hit |= u[j] >= 0 && ((f[j] >> (u[j] & 31)) & 1u);
      if (kCount) bytes += 8LL * min(4u, stop - i);
    }
    for (unsigned rest = __ballot_sync(FULL, !hit && stop < end); rest; rest &= rest - 1) {
      const int l = __ffs(rest) - 1;
      const uint32_t le = __shfl_sync(FULL, end, l);
      bool found = false;
      for (uint32_t p = __shfl_sync(FULL, stop, l); p < le && !found; p += 128) {
        int u[4];
        bool f = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t q = p + 32 * j + lane;
          u[j] = q < le ? __ldg(g.csc_src + q) : -1;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) f |= u[j] >= 0 && ((F[u[j] >> 5] >> (u[j] & 31)) & 1u);
        found = __any_sync(FULL, f);
        if (kCount && lane == l) bytes += 8LL * min(128u, le - p);
      }
      if (lane == l) hit = found;
    }
    if (hit) {
      g.depth[v] = level;
      edges += __ldg(g.csr_off + v + 1) - __ldg(g.csr_off + v);
      ++members;
    }
    const unsigned word = __ballot_sync(FULL, hit);
    if (lane == 0) N[w] = word;
    u0 = b1 < e1 ? __ldg(g.csc_src + b1) : 0;
    b0 = b1;
    e0 = e1;
    d1 = d2;
  }
}

template <bool kCount, bool kCluster>
__global__ void __launch_bounds__(kSbNT, 1)
    k_bfs_small(Bfs g, const int32_t *__restrict__ act, int n_act, uint32_t *bits, Queue qa,
                Queue qb, int nW, long long nE, int forced, int max_iter, SmallCtl *c,
                gas_counters *cnt) {
  // head: the level to expand; a barrier wait that gave up: every CTA leaves,
  // the error goes straight to the engine's counters (the epilogue below
  // does not run)
#define SB_SYNC(out, from)                                                       \
  do {                                                                           \
    const auto load = [&] { return __ldcg(reinterpret_cast<const int4 *>(from)); }; \
    if constexpr (kCluster) {                                                    \
      gasgrid::cluster_barrier_with(&(out), load);                               \
    } else if (!gasgrid::barrier_with(&c->bar, bar, &(out), load)) {             \
      if (threadIdx.x == 0) atomicExch(&cnt->error, (int)GAS_ERR_DEVICE);        \
      return;                                                                    \
    }                                                                            \
  } while (0)
  __shared__ Stage st;
  __shared__ int s_row[kWarps][32][3];
  __shared__ int s_sum[2];
  const int tid = blockIdx.x * kSbNT + threadIdx.x, nthr = gridDim.x * kSbNT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int bar = c->bar.next;
  int4 head;
  long long bytes = 0;
  if (threadIdx.x == 0) st.n = 0;
  __syncthreads();
  // level 0: the active set's unvisited vertices
  for (int i0 = tid - lane; i0 < n_act; i0 += nthr) {
    int v[1] = {i0 + lane < n_act ? __ldg(act + i0 + lane) : -1};
    if (kCount && v[0] >= 0) bytes += 8;
    if (v[0] >= 0 && atomicCAS(g.depth + v[0], -1, 0) == -1) {
      atomicOr(bits + (v[0] >> 5), 1u << (v[0] & 31));
    } else {
      v[0] = -1;
    }
    offer(st, v, g.csr_off, qa, &c->q[0]);
  }
  flush(st, g.csr_off, qa, &c->q[0]);
  SB_SYNC(head, &c->q[0]);
  int it = 1, n_push = 0, n_pull = 0;
  // the cap stays in each CTA: every CTA stops at the same level
  bool capped = false;
  bool pulled = false;    // the frontier was found bottom-up
  bool unqueued = false;  // it is in the bitmap only
  int mk = 0;             // made[mk] is the next made queue's count, and is clear
  long long seen = 0;                   // out-edges of the levels expanded
  int prev = 0;                         // members of the level before
  for (int k = 0;; ++k) {
    const int cur = k % 3, nxt = (k + 1) % 3, old = (k + 2) % 3;
    const int edges = head.z, members = head.w;
    if (edges == 0) break;  // A_{k+1} = N(C_k) is empty
    if (it >= max_iter) {
      capped = true;
      break;
    }
    ++it;
    const int level = k + 1;
    const bool pull =
        forced == 2 ||
        (pulled ? members >= prev || (long long)members * kSbBeta > g.nV
                : (long long)edges * kSbAlpha > nE - seen);
    seen += edges;
    prev = members;
    const uint32_t *F = bits + (size_t)cur * nW;
    uint32_t *N = bits + (size_t)nxt * nW;
    uint32_t *O = bits + (size_t)old * nW;
    // the buffers of level k-1 were last read before the previous barrier
    for (int w = tid; w < nW; w += nthr) O[w] = 0u;
    if (tid == 0) *reinterpret_cast<int4 *>(&c->q[old]) = make_int4(0, 0, 0, 0);
    const Queue Q = k & 1 ? qb : qa, next = k & 1 ? qa : qb;
    if (!pull && unqueued) {  // the queue of a frontier that is in the bitmap only
      Count *made = &c->made[mk];
      for (int w0 = dealt_warp(); w0 < nW; w0 += nthr >> 5) {
        const uint32_t word = F[w0];
        if (!word) continue;  // warp-uniform
        const int v[1] = {(word >> lane) & 1u ? (w0 << 5) + lane : -1};
        offer(st, v, g.csr_off, Q, made);
      }
      flush(st, g.csr_off, Q, made);
      SB_SYNC(head, made);
      // the other count was last read before the barrier that ended its own
      // level, and the one that ends this level comes before it is added to
      // again.  (One count, cleared after the level's end, is being added to
      // by then where the next level makes its queue as well.)
      mk ^= 1;
      if (tid == 0) *reinterpret_cast<int4 *>(&c->made[mk]) = make_int4(0, 0, 0, 0);
    }
    unqueued = pull || edges >= kSbDense * nthr;
    int e = 0, m = 0;  // this level's finds, when they are not queued
    const int w0 = head.y % (nthr / 32);  // light rows begin where the heavy ones end
    if (pull) {
      sb_pull<kCount>(g, F, N, nW, level, e, m, bytes);
    } else if (unqueued) {
      sb_walk<kCount, true>(g, Q.heavy, head.y, kHeavyMost, 0, level, N, s_row[warp], st, next,
                            &c->q[nxt], e, m, bytes);
      sb_walk<kCount, true>(g, Q.light, head.x, 32, w0, level, N, s_row[warp], st, next,
                            &c->q[nxt], e, m, bytes);
    } else {
      sb_walk<kCount, false>(g, Q.heavy, head.y, kHeavyMost, 0, level, N, s_row[warp], st, next,
                             &c->q[nxt], e, m, bytes);
      sb_walk<kCount, false>(g, Q.light, head.x, 32, w0, level, N, s_row[warp], st, next,
                             &c->q[nxt], e, m, bytes);
      flush(st, g.csr_off, next, &c->q[nxt]);
    }
    if (unqueued) {  // one addition per CTA
      if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
      __syncthreads();
      e = __reduce_add_sync(0xffffffffu, e);
      m = __reduce_add_sync(0xffffffffu, m);
      if (lane == 0 && m) {
        atomicAdd(&s_sum[0], e);
        atomicAdd(&s_sum[1], m);
      }
      __syncthreads();
      if (threadIdx.x == 0 && s_sum[1]) {
        atomicAdd(&c->q[nxt].edges, s_sum[0]);
        atomicAdd(&c->q[nxt].members, s_sum[1]);
      }
    }
    pulled = pull;
    if (pull)
      ++n_pull;
    else
      ++n_push;
    SB_SYNC(head, &c->q[nxt]);
  }
  if (kCount) warp_add(bytes, &c->bytes);
  // the next run finds the bitmaps clear (nothing reads them any more)
  for (int w = tid; w < 3 * nW; w += nthr) bits[w] = 0u;
  if (tid == 0) {
    // the engine's counters, as the fast schedule leaves them
    cnt->iteration = it;
    cnt->n_push = n_push;
    cnt->n_pull = n_pull;
    cnt->error = capped ? GAS_ERR_ITER_CAP : 0;
    if (!capped) cnt->n_active = 0;
    c->bar.next = bar;
    // and the control word clear for the next run (a CTA still to read a
    // count finds no edges and leaves as well)
    c->q[0] = c->q[1] = c->q[2] = Count{0, 0, 0, 0};
    c->made[0] = c->made[1] = Count{0, 0, 0, 0};
  }
#undef SB_SYNC
}

}  // namespace

namespace gas {

cudaError_t launch_small(void *grid_fn, void *cluster_fn, int cluster_upto, const gas_engine *e,
                         void **args, cudaStream_t s) {
  const int64_t want = std::max<int64_t>(1, ((int64_t)e->nV + e->nE) / kCtaEdges);
  if (want <= cluster_upto) {
    const int n = (int)std::min<int64_t>(want, kClusterMost);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = n;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n);
    cfg.blockDim = dim3(kNT);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaError_t ce = n > 8 ? cudaFuncSetAttribute(
                                 cluster_fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)
                           : cudaSuccess;
    if (ce == cudaSuccess) ce = cudaLaunchKernelExC(&cfg, cluster_fn, args);
    if (ce == cudaSuccess) return ce;
    cudaGetLastError();  // no room for such a cluster: a cooperative grid
  }
  return cudaLaunchCooperativeKernel(grid_fn, dim3((int)std::min<int64_t>(want, e->num_sms)),
                                     dim3(kNT), args, 0, s);
}

bool bfs_small_eligible(const gas_engine *e, gas_schedule_t schedule) {
  const char *v = getenv("GAS_BFS_SMALL");
  if (v && v[0] == '0') return false;
  // PUSH forces the multi-kernel loop's kernels
  if (e->prog != GAS_PROG_BFS || schedule == GAS_SCHED_PUSH || e->edges_on_host) return false;
  // per-iteration records, and on all but small graphs the split of the time
  // by direction, come from the multi-kernel loop
  if (e->nV > kBfsSmallRecordsMaxV && (e->trace_on || e->profiling)) return false;
  return e->nV <= kBfsSmallMaxV && e->nV > 0;
}

SmallBytes bfs_small_bytes(int64_t nV, int64_t nE) {
  return {(size_t)(3 * ((nV + 31) / 32)) * sizeof(uint32_t), sizeof(SmallCtl),
          2 * ((size_t)nV + heavy_cap(nE)) * sizeof(int4)};
}

bool bfs_small_reserve(gas_engine *e) {
  if (e->sb_bits) return true;
  const SmallBytes n = bfs_small_bytes(e->nV, e->nE);
  e->sb_clean = false;
  if (e->sb_mem.alloc({GROUP_PART(e->sb_bits, n.values), GROUP_PART(e->sb_ctl, n.ctl),
                       GROUP_PART(e->sb_queue, n.queues)}) == cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}

gas_status_t run_bfs_small(gas_engine *e, gas_schedule_t schedule, int32_t max_iterations,
                           gas_run_stats *stats, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const int nW = (e->nV + 31) / 32;
  const size_t V = (size_t)e->nV, H = heavy_cap(e->nE);
  SmallCtl *ctl = static_cast<SmallCtl *>(e->sb_ctl);
  const bool count = e->profiling;
  // the kernel leaves its bitmaps and control word clear; they are cleared
  // here after allocation, after a run that failed, and when bytes count
  if (!e->sb_clean || count) {
    CUDA_TRY(cudaMemsetAsync(e->sb_bits, 0, (size_t)3 * nW * sizeof(uint32_t), s));
    CUDA_TRY(cudaMemsetAsync(ctl, 0, sizeof(SmallCtl), s));
  }
  e->sb_clean = false;
  gas_counters *cnt = e->cnt;
  Bfs g{e->csr_off, e->csr_dst, e->csc_off, e->csc_src, static_cast<int32_t *>(e->vd), e->nV};
  const int32_t *act = e->act;
  int n_act = e->n_active, nw = nW;
  uint32_t *bits = e->sb_bits;
  int4 *q = static_cast<int4 *>(e->sb_queue);
  Queue qa{q, q + V}, qb{q + V + H, q + 2 * V + H};
  long long nE = e->nE;
  int forced = schedule == GAS_SCHED_PULL ? 2 : 0;
  int max_iter = max_iterations;
  void *args[] = {&g, &act, &n_act, &bits, &qa, &qb, &nw, &nE, &forced, &max_iter, &ctl, &cnt};
  if (count) prof_begin(e, s, kProfPush, 0);
  void *grid_fn = count ? (void *)k_bfs_small<true, false> : (void *)k_bfs_small<false, false>;
  void *cluster_fn = count ? (void *)k_bfs_small<true, true> : (void *)k_bfs_small<false, true>;
  CUDA_TRY(launch_small(grid_fn, cluster_fn, kSbCluster, e, args, s));
  prof_end(e, s);
  if (count) {
    SmallCtl h;
    CUDA_TRY(cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    e->prof_bytes_pending = h.bytes;
    prof_collect(e);
  }
  gas_counters c;
  GAS_TRY(engine_sync_counts(e, stream));
  c = *e->h_cnt;
  e->sb_clean = c.error == 0 || c.error == GAS_ERR_ITER_CAP;
  if (stats) {
    stats->iterations = c.iteration;
    stats->push_iters = c.n_push;
    stats->pull_iters = c.n_pull;
    stats->kernel_launches = 1;
    stats->graph_launches = 0;
  }
  e->level = c.iteration;
  e->active_full = false;
  return loop_status(e, c, stream);
}

}  // namespace gas
