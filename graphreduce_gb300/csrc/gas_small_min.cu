// gas_small_min.cu -- SSSP and CC on small and medium graphs as one
// persistent kernel.
//
// An iteration of the fast schedule is a WHILE round of six kernel nodes, 25
// to 40 us however little there is to do.  Here one cooperative launch runs
// every iteration as a push, from the full active set: the same changed sets
// C_k, vertex data and iteration count as run() (gas_sched.cu states why a
// push from C_k equals a pull over the active set).
//
//   values       two buffers.  Iteration k reads R (the values at its start,
//                which nothing writes during it: bulk-synchronous, and plain
//                L1-cached loads are exact) and lowers W with atomicMin; the
//                two then swap.  At its start W equals R but for the members
//                of C_k, lowered in the iteration before: each member's
//                queue entry also does atomicMin(W[u], R[u]).
//   sparse       v joins the next queue when a candidate below R[v] is the
//                first to lower W[v]: the first atomicMin to get there finds
//                a value >= R[v] (R[v] itself, or the older one if v is in
//                C_k and not yet copied), every later one a value below
//                R[v].  One returning atomic per lowering candidate, no
//                bitmap, no compaction pass, one grid barrier.
//   dense        (kDense or more out-edges per thread of the grid) the
//                candidates only lower W, with reductions nobody waits for;
//                after a second barrier the members are the vertices with
//                W[v] < R[v], found by one coalesced pass.
//   queue        a CTA collects its new members in shared memory and appends
//                them to the global queue after its edges: light members as
//                one entry each, the others as entries of kEntryEdges edges
//                (a hub is many entries, so any run of entries is balanced);
//                members without out-edges are light entries, for the copy
//                into W.
//   walk         a warp takes some consecutive entries, as many as spread
//                them over all warps, and walks their edges laid end to end,
//                four rounds of 32 in flight.
//
// Small queues are bound by the latency of the chain entry -> value -> edge
// -> target -> atomic -> append -> barrier, about 6 us; the grid has a CTA
// per kCtaEdges vertices and edges, at most one per SM, as a barrier among
// fewer CTAs is cheaper.  Big ones by L2 lookups (a random value per edge).
// Measured against the fast schedule (us per run, SSSP, AUTO / LEARNED /
// here): R-MAT 16 edges per vertex, 4,093 vertices 389 / 356 / 106, 262 K
// 557 / 459 / 256, 1 M 1365 / 743 / 597, 2 M 1787 / 978 / 901, 4 M 3747 /
// 1756 / 1810; Erdos-Renyi 12 per vertex, 65 K 736 / 744 / 242, 1 M 2385 /
// 1532 / 1020, 2 M 4414 / 2367 / 2092.  CC on R-MAT, 65 K 285 / 265 / 119,
// 1 M 958 / 492 / 459, 2 M 1561 / 731 / 824, 4 M 2741 / 1358 / 1510.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "gas.h"
#include "gas_engine_impl.h"
#include "gas_internal.h"
#include "gas_sched.h"
#include "gas_stage.cuh"

namespace {

using namespace gasstage;

constexpr int kMinCluster = 32;   // CTAs asked for up to which a cluster is enough (R-MAT
                                  // 4 K, 60 CTAs: 117 us against 113)
constexpr int kDense = 8;         // 2: 4 % slower on Erdos-Renyi 65 K, even on R-MAT

struct MinCtl {
  gasgrid::Barrier bar;
  Count q[3];  // of the queue being read, filled and cleared (rotating)
};

// One warp's share of a queue's light or heavy entries: up to 32 at a time,
// as many as spread them over all warps, beginning with warp w0.
// kLowerOnly: a reduction per candidate below W's value (stale at worst, and
// then above); the members are found afterwards.  Otherwise each first
// lowering offers its target.
template <bool kWeighted, bool kLowerOnly>
__device__ __forceinline__ void walk(const int4 *Q, int nq, int most, int w0,
                                     const int32_t *R, int32_t *W, const int32_t *csr_off,
                                     const int32_t *csr_dst, const int32_t *csr_w,
                                     int32_t zero_cap, int (*s_row)[3], Stage &st,
                                     const Queue &N, Count *ctr) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kRounds = 4;
  const int lane = threadIdx.x & 31;
  const int nwarps = gridDim.x * kWarps;
  int gwarp = dealt_warp() - w0;
  if (gwarp < 0) gwarp += nwarps;
  const int per = min(most, (nq + nwarps - 1) / nwarps);
  for (long long base = (long long)gwarp * per; base < nq; base += (long long)nwarps * per) {
    int start = 0, deg = 0, val = 0;
    if (lane < per && base + lane < nq) {
      const int4 e = Q[base + lane];
      start = e.y;
      deg = e.z;
      val = R[e.x];
      atomicMin(W + e.x, val);
    }
    Rows rows;
    const int T = lay_out(start, deg, val, s_row, rows);
    for (int r = 0; r < T; r += 32 * kRounds) {
      int v[kRounds], cand[kRounds], cur[kRounds];
#pragma unroll
      for (int h = 0; h < kRounds; ++h) {
        const int r0 = r + 32 * h;
        const int row = row_of(rows, r0);
        const int pos = r0 + lane + __shfl_sync(FULL, rows.shift, row);
        cand[h] = __shfl_sync(FULL, rows.val, row);
        v[h] = -1;
        if (r0 + lane < T) {
          v[h] = ld_edge(csr_dst + pos);
          if (kWeighted) cand[h] += ld_edge(csr_w + pos);
        }
      }
#pragma unroll
      for (int h = 0; h < kRounds; ++h) {
        cand[h] = min(cand[h], zero_cap);
        cur[h] = v[h] < 0 ? INT_MIN : kLowerOnly ? W[v[h]] : R[v[h]];
      }
      if constexpr (kLowerOnly) {
#pragma unroll
        for (int h = 0; h < kRounds; ++h)
          if (cand[h] < cur[h]) atomicMin(W + v[h], cand[h]);
      } else {
        int old[kRounds];
#pragma unroll
        for (int h = 0; h < kRounds; ++h) {
          old[h] = INT_MIN;
          if (cand[h] < cur[h]) old[h] = atomicMin(W + v[h], cand[h]);
        }
#pragma unroll
        for (int h = 0; h < kRounds; ++h)
          if (!(cand[h] < cur[h] && old[h] >= cur[h])) v[h] = -1;  // not the first to lower it
        offer(st, v, csr_off, N, ctr);
      }
    }
  }
}

template <bool kWeighted, bool kCluster>
__global__ void __launch_bounds__(kNT, 1)
    k_min_small(const int32_t *__restrict__ csr_off, const int32_t *__restrict__ csr_dst,
                const int32_t *__restrict__ csr_w, int32_t *vd, int32_t *vd2, Queue qa, Queue qb,
                int nV, int32_t zero_cap, int max_iter, MinCtl *c, gas_counters *cnt) {
  // head: the queue to read next; a barrier wait that gave up: every CTA
  // leaves
#define MIN_SYNC(next)                                                            \
  do {                                                                            \
    const auto load = [&] {                                                       \
      return __ldcg(reinterpret_cast<const int4 *>(&c->q[(next) % 3]));           \
    };                                                                            \
    if constexpr (kCluster) {                                                     \
      gasgrid::cluster_barrier_with(&head, load);                                 \
    } else if (!gasgrid::barrier_with(&c->bar, bar, &head, load)) {               \
      if (threadIdx.x == 0) atomicExch(&cnt->error, (int)GAS_ERR_DEVICE);         \
      return;                                                                     \
    }                                                                             \
  } while (0)
  __shared__ Stage st;
  __shared__ int s_row[kWarps][32][3];  // excl, CSR position - excl, value
  const int tid = blockIdx.x * kNT + threadIdx.x, nthr = gridDim.x * kNT;
  const int warp = threadIdx.x >> 5;
  unsigned int bar = c->bar.next;
  int4 head;
  if (threadIdx.x == 0) st.n = 0;
  __syncthreads();
  // C_{-1}: only values below Program::gatherZero can lower anything
  for (int v0 = blockIdx.x * kStage; v0 < nV; v0 += gridDim.x * kStage) {
#pragma unroll
    for (int i = 0; i < kStage; i += kNT) {
      const int v = v0 + i + threadIdx.x;
      int x = INT_MAX;
      if (v < nV) vd2[v] = x = vd[v];
      const int in[1] = {x < zero_cap ? v : -1};
      offer(st, in, csr_off, qa, &c->q[0]);
    }
    flush(st, csr_off, qa, &c->q[0]);
  }
  MIN_SYNC(0);
  int it = 0;
  bool capped = false;
  int edges = 0;
  for (int k = 0;; ++k) {
    edges = head.z;
    if (k > 0 && edges == 0) break;  // A_{k+1} = N(C_k) is empty
    if (it >= max_iter) {            // every CTA stops here at the same iteration
      capped = true;
      break;
    }
    ++it;
    const int32_t *R = k & 1 ? vd2 : vd;
    int32_t *W = k & 1 ? vd : vd2;
    const Queue Q = k & 1 ? qb : qa, N = k & 1 ? qa : qb;
    Count *ctr = &c->q[(k + 1) % 3];
    if (tid == 0)  // last read before the previous barrier
      *reinterpret_cast<int4 *>(&c->q[(k + 2) % 3]) = make_int4(0, 0, 0, 0);
    const int w0 = head.y % (nthr / 32);  // light rows begin where the heavy ones end
    if (edges < kDense * nthr) {
      walk<kWeighted, false>(Q.heavy, head.y, kHeavyMost, 0, R, W, csr_off, csr_dst, csr_w,
                             zero_cap, s_row[warp], st, N, ctr);
      walk<kWeighted, false>(Q.light, head.x, 32, w0, R, W, csr_off, csr_dst, csr_w, zero_cap,
                             s_row[warp], st, N, ctr);
      flush(st, csr_off, N, ctr);
    } else {
      walk<kWeighted, true>(Q.heavy, head.y, kHeavyMost, 0, R, W, csr_off, csr_dst, csr_w, zero_cap,
                            s_row[warp], st, N, ctr);
      walk<kWeighted, true>(Q.light, head.x, 32, w0, R, W, csr_off, csr_dst, csr_w, zero_cap,
                            s_row[warp], st, N, ctr);
      MIN_SYNC(k);
      // the members: every vertex whose value fell
      for (int v0 = blockIdx.x * kStage; v0 < nV; v0 += gridDim.x * kStage) {
#pragma unroll
        for (int i = 0; i < kStage; i += kNT) {
          const int v = v0 + i + threadIdx.x;
          const int in[1] = {v < nV && W[v] < R[v] ? v : -1};
          offer(st, in, csr_off, N, ctr);
        }
        flush(st, csr_off, N, ctr);
      }
    }
    MIN_SYNC(k + 1);
  }
  // the values are in the buffer the last iteration wrote
  if (it & 1)
    for (int v = tid; v < nV; v += nthr) vd[v] = vd2[v];
  if (tid == 0) {
    // the engine's counters, as the fast schedule leaves them
    cnt->iteration = it;
    cnt->n_push = it;
    cnt->n_pull = 0;
    cnt->n_scatter_edges = edges;
    cnt->cond = 0;
    cnt->error = capped ? GAS_ERR_ITER_CAP : 0;
    if (!capped) cnt->n_active = 0;
    c->bar.next = bar;
    // and the queue counters clear for the next run (a CTA still to read one
    // finds no edges and leaves as well)
    c->q[0] = c->q[1] = c->q[2] = Count{0, 0, 0, 0};
  }
#undef MIN_SYNC
}

}  // namespace

namespace gas {

bool min_small_eligible(const gas_engine *e, gas_schedule_t schedule) {
  if (e->prog != GAS_PROG_SSSP && e->prog != GAS_PROG_CC) return false;
  // PUSH and PULL force the multi-kernel loop's kernels.  LEARNED has the
  // head's choices to lose where the multi-kernel push is as fast
  if (schedule != GAS_SCHED_AUTO && schedule != GAS_SCHED_LEARNED) return false;
  // per-iteration records and kernel times come from the multi-kernel loop
  if (e->trace_on || e->profiling || e->edges_on_host) return false;
  if (!e->active_full || e->counts_dirty || e->n_active != e->nV) return false;
  const int learned =
      e->prog == GAS_PROG_SSSP ? kSsspSmallLearnedMaxV : kCcSmallLearnedMaxV;
  return e->nV > 0 && e->nV <= (schedule == GAS_SCHED_AUTO ? kMinSmallMaxV : learned);
}

SmallBytes min_small_bytes(int64_t nV, int64_t nE) {
  return {(size_t)nV * sizeof(int32_t), sizeof(MinCtl),
          2 * ((size_t)nV + heavy_cap(nE)) * sizeof(int4)};
}

bool min_small_reserve(gas_engine *e) {
  if (e->sm_vals) return true;
  const SmallBytes n = min_small_bytes(e->nV, e->nE);
  e->sm_clean = false;
  if (e->sm_mem.alloc({GROUP_PART(e->sm_vals, n.values), GROUP_PART(e->sm_ctl, n.ctl),
                       GROUP_PART(e->sm_queue, n.queues)}) == cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}

gas_status_t run_min_small(gas_engine *e, int32_t max_iterations, gas_run_stats *stats,
                           void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const size_t V = (size_t)e->nV, H = heavy_cap(e->nE);
  // the kernel leaves its control word clear; cleared here at first and
  // after a run that failed
  if (!e->sm_clean) CUDA_TRY(cudaMemsetAsync(e->sm_ctl, 0, sizeof(MinCtl), s));
  e->sm_clean = false;
  const bool weighted = e->prog == GAS_PROG_SSSP;
  const int32_t *csr_off = e->csr_off, *csr_dst = e->csr_dst;
  const int32_t *csr_w = static_cast<const int32_t *>(e->csr_ed);
  int32_t *vd = static_cast<int32_t *>(e->vd), *vd2 = e->sm_vals;
  int4 *q = static_cast<int4 *>(e->sm_queue);
  Queue qa{q, q + V}, qb{q + V + H, q + 2 * V + H};
  int nV = e->nV;
  int32_t zero_cap = weighted ? INT_MAX - 100000 : INT_MAX;
  MinCtl *ctl = static_cast<MinCtl *>(e->sm_ctl);
  gas_counters *cnt = e->cnt;
  void *args[] = {&csr_off, &csr_dst, &csr_w, &vd, &vd2, &qa, &qb, &nV, &zero_cap,
                  &max_iterations, &ctl, &cnt};
  void *grid_fn =
      weighted ? (void *)k_min_small<true, false> : (void *)k_min_small<false, false>;
  void *cluster_fn =
      weighted ? (void *)k_min_small<true, true> : (void *)k_min_small<false, true>;
  CUDA_TRY(launch_small(grid_fn, cluster_fn, kMinCluster, e, args, s));
  GAS_TRY(engine_sync_counts(e, stream));
  const gas_counters c = *e->h_cnt;
  e->sm_clean = c.error == 0 || c.error == GAS_ERR_ITER_CAP;
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
