// gas_runs.cu -- whole-algorithm runs on a device-resident graph:
//   * gas_engine_run_schedule: run() (gpugas.h:1792-1807) with the loop moved
//     onto the device -- one iteration's kernels are captured once into the
//     body of a CUDA-graph WHILE node whose condition a tiny kernel sets from
//     the device counters, so there is no host round trip per iteration;
//   * gas_engine_pagerank_precision: the normalised PageRank with FP32
//     compensated (two-sum) gather and an FP64 L1 residual deciding
//     convergence on the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "gas.h"
#include "gas_device.cuh"
#include "gas_engine_impl.h"
#include "gas_internal.h"
#include "gas_sched.h"

using gasdev::kNT;
using gasdev::SegSource;

namespace {

inline cudaStream_t S(void *s) { return (cudaStream_t)s; }

__global__ void k_reset_loop(gas_counters *cnt, int32_t max_iter) {
  cnt->iteration = 0;
  cnt->error = 0;
  cnt->cond = 1;
  cnt->max_iter = max_iter;
}

}  // namespace

namespace gas {

// Builds graph = WHILE(cond) { body(stream, handle) } and instantiates it.
gas_status_t build_while_graph(
    gas_engine *e,
    gas_status_t (*body)(gas_engine *, cudaStream_t, cudaGraphConditionalHandle,
                         void *),
    void *ctx, cudaGraphExec_t *out) {
  cudaGraph_t g = nullptr;
  cudaStream_t cs = nullptr;
  cudaGraphExec_t x = nullptr;
  gas_status_t st = GAS_OK;
  cudaGraphConditionalHandle h;
  cudaGraphNodeParams p = {};
  cudaGraphNode_t node;
  cudaGraph_t bodyg;
  CUDA_TRY(cudaGraphCreate(&g, 0));
  cudaError_t ce = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault);
  if (ce == cudaSuccess) {
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    ce = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &p);
  }
  if (ce == cudaSuccess) ce = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (ce != cudaSuccess) {
    cudaGraphDestroy(g);
    return fail(GAS_ERR_CUDA, "while-graph setup: %s", cudaGetErrorString(ce));
  }
  bodyg = p.conditional.phGraph_out[0];
  ce = cudaStreamBeginCaptureToGraph(cs, bodyg, nullptr, nullptr, 0,
                                     cudaStreamCaptureModeRelaxed);
  if (ce == cudaSuccess) {
    e->capturing = true;
    e->in_graph = true;
    st = body(e, cs, h, ctx);
    e->capturing = false;
    e->in_graph = false;
    cudaGraph_t captured = nullptr;
    cudaError_t ce2 = cudaStreamEndCapture(cs, &captured);
    if (st == GAS_OK && ce2 != cudaSuccess)
      st = fail(GAS_ERR_CUDA, "end capture: %s", cudaGetErrorString(ce2));
  } else {
    st = fail(GAS_ERR_CUDA, "begin capture: %s", cudaGetErrorString(ce));
  }
  if (st == GAS_OK) {
    ce = cudaGraphInstantiate(&x, g, 0);
    if (ce != cudaSuccess)
      st = fail(GAS_ERR_CUDA, "instantiate: %s", cudaGetErrorString(ce));
  }
  cudaStreamDestroy(cs);
  cudaGraphDestroy(g);
  if (st == GAS_OK) *out = x;
  return st;
}

bool host_loop_requested() {
  const char *v = getenv("GAS_HOST_LOOP");
  return v && v[0] == '1';
}

bool host_loop_for(const gas_engine *e) {
  return e->profiling || host_loop_requested();
}

// The same loop without a graph: body launches on the stream, the host
// reads the condition word after every iteration.
gas_status_t run_host_loop(
    gas_engine *e,
    gas_status_t (*body)(gas_engine *, cudaStream_t, cudaGraphConditionalHandle,
                         void *),
    void *ctx, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  gas_status_t st = GAS_OK;
  e->capturing = true;
  e->in_graph = false;
  for (;;) {
    cudaError_t ce = cudaMemcpyAsync(e->h_cnt, e->cnt, sizeof(gas_counters),
                                     cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (ce != cudaSuccess) {
      st = fail(GAS_ERR_CUDA, "host loop: %s", cudaGetErrorString(ce));
      break;
    }
    if (!e->h_cnt->cond) break;
    st = body(e, s, 0, ctx);
    if (st != GAS_OK) break;
    prof_collect(e);
  }
  e->capturing = false;
  return st;
}

// Turns the device error word / a non-empty frontier after the loop into a
// status, and clears the word so the engine stays usable.
gas_status_t loop_status(gas_engine *e, const gas_counters &c, void *stream) {
  if (c.error)
    CUDA_TRY(cudaMemsetAsync(&e->cnt->error, 0, sizeof(int32_t), S(stream)));
  if (c.error == GAS_ERR_ITER_CAP || (c.error == 0 && c.n_active > 0))
    return fail(GAS_ERR_ITER_CAP, "no convergence within %d iterations", c.iteration);
  if (c.error)
    return fail(GAS_ERR_DEVICE, "device error word %d after %d iterations", c.error,
                c.iteration);
  return GAS_OK;
}

}  // namespace gas

namespace {

struct GenericCtx {
  bool ordered;
};

gas_status_t generic_body(gas_engine *e, cudaStream_t cs,
                          cudaGraphConditionalHandle h, void *ctx) {
  const GenericCtx *c = static_cast<const GenericCtx *>(ctx);
  return gas::engine_generic_iteration(e, c->ordered, h, cs);
}

}  // namespace

extern "C" gas_status_t gas_engine_run_schedule(gas_engine *e,
                                                gas_schedule_t schedule,
                                                int32_t max_iterations,
                                                gas_run_stats *stats,
                                                void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "run before set_graph");
  if (e->prog == GAS_PROG_USER)
    return gas::fail(GAS_ERR_UNSUPPORTED, "user programs run through gpugas.h");
  // default cap: nV + 2 bounds every correct BFS / SSSP / CC run (each
  // iteration settles at least one more vertex); PageRank gets 100000
  if (max_iterations <= 0)
    max_iterations = e->prog == GAS_PROG_PAGERANK ? 100000 : e->nV + 2;
  if (stats) *stats = gas_run_stats{};
  int32_t n = 0;
  GAS_TRY(gas_engine_count_active(e, &n));
  if (e->pending_gather || e->slots_pending)
    return gas::fail(GAS_ERR_STATE, "run_schedule in the middle of a step");
  if (n == 0) return GAS_OK;
  if (schedule != GAS_SCHED_GENERIC && schedule != GAS_SCHED_ORDERED)
    return gas::run_fast(e, schedule, max_iterations, stats, stream);

  GenericCtx ctx{schedule == GAS_SCHED_ORDERED};
  const bool gathers = e->prog != GAS_PROG_BFS && !ctx.ordered;
  if (gathers) GAS_TRY(gas::engine_partition(e, stream));  // the first iteration's
  const int slot = ctx.ordered ? kGraphOrdered : kGraphGeneric;
  if (gas::host_loop_for(e)) {
    k_reset_loop<<<1, 1, 0, S(stream)>>>(e->cnt, max_iterations);
    CUDA_TRY(cudaGetLastError());
    e->level_from_counters = true;
    gas_status_t st = gas::run_host_loop(e, generic_body, &ctx, stream);
    e->level_from_counters = false;
    if (st != GAS_OK) return st;
  } else {
  if (!e->graphs[slot]) {
    e->level_from_counters = true;
    gas_status_t st = gas::build_while_graph(e, generic_body, &ctx, &e->graphs[slot]);
    e->level_from_counters = false;
    if (st != GAS_OK) return st;
  }
  k_reset_loop<<<1, 1, 0, S(stream)>>>(e->cnt, max_iterations);
  cudaError_t ce = cudaGetLastError();
  if (ce == cudaSuccess) ce = cudaGraphLaunch(e->graphs[slot], S(stream));
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(S(stream));
  if (ce != cudaSuccess)
    return gas::fail(GAS_ERR_CUDA, "generic run: %s", cudaGetErrorString(ce));
  }
  gas_counters c;
  GAS_TRY(gas_engine_read_counters(e, &c, stream));
  if (stats) {
    stats->iterations = c.iteration;
    // per iteration: gather tiles + fixup (ordered: one kernel; BFS: apply),
    // commit + expansion in two, compaction in two or three, the last of
    // them also the loop condition; plus the reset and the first partition
    stats->kernel_launches =
        c.iteration * ((gathers ? 2 : 1) + gas::engine_scatter_kernels(e)) + (gathers ? 2 : 1);
    stats->graph_launches = gas::host_loop_for(e) ? 0 : 1;
  }
  e->level = c.iteration;
  e->active_full = false;
  return gas::loop_status(e, c, stream);
}

// ---------------------------------------------------------------------------
// run() of a user program: the Program-typed kernels come from the caller's
// translation unit through a step callback; the rest of the iteration is
// libgas's, and the loop is a WHILE node on the device.
// ---------------------------------------------------------------------------
namespace {

struct UserCtx {
  gas_user_step_fn step;
  void *ctx;
  int32_t wrote_slots;
};

gas_status_t user_body(gas_engine *e, cudaStream_t cs, cudaGraphConditionalHandle h,
                       void *ctx) {
  const UserCtx *u = static_cast<const UserCtx *>(ctx);
  GAS_TRY(u->step(u->ctx, cs));
  CUDA_TRY(cudaGetLastError());
  e->slots_pending = u->wrote_slots != 0;
  return gas::engine_scatter_loop(e, h, cs);
}

}  // namespace

extern "C" gas_status_t gas_engine_run_user(gas_engine *e, gas_user_step_fn step,
                                            void *ctx, int32_t wrote_slots,
                                            int32_t max_iterations, gas_run_stats *stats,
                                            void *stream) {
  if (!e || !step) return gas::fail(GAS_ERR_INVALID, "run_user: null argument");
  if (!e->has_graph) return gas::fail(GAS_ERR_STATE, "run before set_graph");
  if (e->prog != GAS_PROG_USER)
    return gas::fail(GAS_ERR_UNSUPPORTED, "run_user: built-in programs use run_schedule");
  if (max_iterations <= 0) max_iterations = 1000000;
  if (stats) *stats = gas_run_stats{};
  int32_t n = 0;
  GAS_TRY(gas_engine_count_active(e, &n));
  if (e->pending_gather || e->slots_pending)
    return gas::fail(GAS_ERR_STATE, "run_user in the middle of a step");
  if (n == 0) return GAS_OK;
  UserCtx u{step, ctx, wrote_slots != 0 ? 1 : 0};
  const bool direct = gas::host_loop_for(e);
  if (direct) {
    k_reset_loop<<<1, 1, 0, S(stream)>>>(e->cnt, max_iterations);
    CUDA_TRY(cudaGetLastError());
    GAS_TRY(gas::run_host_loop(e, user_body, &u, stream));
  } else {
    if (e->graphs[kGraphUser] && (e->user_step != step || e->user_ctx != ctx ||
                                  e->user_wrote_slots != u.wrote_slots)) {
      cudaGraphExecDestroy(e->graphs[kGraphUser]);
      e->graphs[kGraphUser] = nullptr;
    }
    if (!e->graphs[kGraphUser]) {
      GAS_TRY(gas::build_while_graph(e, user_body, &u, &e->graphs[kGraphUser]));
      e->user_step = step;
      e->user_ctx = ctx;
      e->user_wrote_slots = u.wrote_slots;
    }
    k_reset_loop<<<1, 1, 0, S(stream)>>>(e->cnt, max_iterations);
    cudaError_t ce = cudaGetLastError();
    if (ce == cudaSuccess) ce = cudaGraphLaunch(e->graphs[kGraphUser], S(stream));
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(S(stream));
    if (ce != cudaSuccess)
      return gas::fail(GAS_ERR_CUDA, "user run: %s", cudaGetErrorString(ce));
  }
  gas_counters c;
  GAS_TRY(gas_engine_read_counters(e, &c, stream));
  if (stats) {
    stats->iterations = c.iteration;
    // per iteration: the caller's partition, tiles and fixup, then commit +
    // expansion and compaction with the loop condition; reset
    stats->kernel_launches = (3 + gas::engine_scatter_kernels(e)) * c.iteration + 1;
    stats->graph_launches = direct ? 0 : 1;
  }
  e->level = c.iteration;
  e->active_full = false;
  return gas::loop_status(e, c, stream);
}

// ---------------------------------------------------------------------------
// Precision-form PageRank.
// ---------------------------------------------------------------------------
namespace {

struct PrVal {
  float s, c;
};

// Error-free transformation: a.s + b.s = s + err exactly (Knuth two-sum);
// compensation terms are carried in c.
__device__ __forceinline__ PrVal two_sum_add(const PrVal &a, const PrVal &b) {
  const float s = __fadd_rn(a.s, b.s);
  const float bp = __fsub_rn(s, a.s);
  const float err = __fadd_rn(__fsub_rn(a.s, __fsub_rn(s, bp)), __fsub_rn(b.s, bp));
  return PrVal{s, __fadd_rn(__fadd_rn(a.c, b.c), err)};
}

// The row epilogue of the precision PageRank: the gathered sum (value +
// compensation) of a destination row becomes its new rank and contribution;
// the L1 step accumulates per thread.
struct PrPol {
  typedef PrVal Val;
  const int32_t *csc_src;
  const float *inv_deg;  // RN(1 / out-degree), 0 without out-edges
  const float *contrib;
  const float *rank_old;
  float *rank_new;
  float *contrib_new;
  float base;       // (1-d)/N, every vertex (seed < 0)
  float base_seed;  // (1-d), the seed only (personalized)
  float damping;
  const int32_t *seed_p;
  int32_t seed;
  double l1;
  // inv and old: the row's reciprocal out-degree and previous rank
  __device__ __forceinline__ void emit(int v, const Val &g, float inv, float old) {
    const float sum = __fadd_rn(g.s, g.c);
    const float b = seed < 0 ? base : (v == seed ? base_seed : 0.0f);
    const float r = __fadd_rn(b, __fmul_rn(damping, sum));
    rank_new[v] = r;
    contrib_new[v] = __fmul_rn(r, inv);
    // the step in FP32 (exact while the two ranks are within a factor of
    // two of each other, Sterbenz), the sum in FP64
    l1 += (double)fabsf(__fsub_rn(r, old));
  }
  __device__ __forceinline__ void emit(int v, const Val &g) {
    emit(v, g, __ldg(inv_deg + v), rank_old[v]);
  }
};

struct PrBufs {
  float *rank[2];
  float *contrib[2];
};

__device__ __forceinline__ void pr_bind(PrPol &pol, const PrBufs &b,
                                        const gas_counters *cnt) {
  const int p = cnt->iteration & 1;
  pol.contrib = b.contrib[p];
  pol.rank_old = b.rank[p];
  pol.rank_new = b.rank[p ^ 1];
  pol.contrib_new = b.contrib[p ^ 1];
  pol.seed = *pol.seed_p;
  pol.l1 = 0.0;
}

__device__ __forceinline__ void block_sum_store(double v, double *out) {
  __shared__ double s_w[32];
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) t += s_w[w];
    *out = t;
  }
}

// ---- gather ----
// A warp owns a tile of kPrW consecutive in-edges, a lane kPrK of them; the
// warps of a CTA never wait for one another.  A tile stages the gathered
// contributions in the warp's shared memory (coalesced index loads, kPrK
// independent gathers per lane), each lane sums its edges sequentially, with
// a bit per edge telling where a row ends, a segmented warp scan of the
// lanes' open-row partials joins rows that span lanes, and the rows that
// start and end inside the tile are finished there with coalesced accesses.
// A row that spans tiles leaves its first part as the tile's tail record and
// the following parts as head records; k_pr_join joins them.  Rows are the
// ones with in-edges (ne_vid); the others' ranks settle in two iterations.
//
// Bound by the L1 data pipe: a wavefront per random contribution (fewer where
// neighbours in a sorted row share a line) and the staging's.  So a row's end
// is a bit, not an item of a merge path with its offset in shared memory and
// a search per lane: 400 instructions a tile where 256 items of the merge
// path took 610, 12 M shared wavefronts where they took 22 M (R-MAT 4 M).
// Measured, ms per run of 45 to 51 iterations, merge path / row-end bits:
// R-MAT 1 M, 8 edges per vertex 2.80 / 2.48, 4 M, 16 per vertex 14.97 /
// 13.12, 16.8 M directed 58.5 / 52.8; with the hot sources below 2.48, 11.3,
// 47.3.
constexpr int kPrK = 8;
constexpr int kPrCtas = 4;
constexpr int kPrCtasMost = 8;     // gather CTAs per SM, and with the join's, which
constexpr int kPrPartsPerSm = 24;  // each leave a part of the residual
constexpr int kPrW = 32 * kPrK;
// s_val is padded by one word per kPrK: a lane reads about kPrK words past
// its neighbour, which without the pad puts 32 / kPrK lanes on one bank
__device__ __forceinline__ int pr_pad(int j) { return j + j / kPrK; }
constexpr int kPrValWords = kPrW + kPrW / kPrK;

// A warp's staging: contributions, sums of the rows that end in the tile.
struct PrStage {
  float val[kPrValWords];
  float sum[kPrW];
};

// Hot sources: the contributions of the kHotSlots sources with the most
// out-edges are copied into each CTA's shared memory, where 32 of them take
// about 3 wavefronts and not up to 32.  A copy of the in-edges, made once per
// graph, has their slots.  163 KB of shared memory with the staging of 32
// warps, for L1 has to hold the lines in flight: with 227 KB (45,000 slots)
// R-MAT 16.8 M took 98 ms, with 99 KB 48.4, with 163 KB 47.3; without hot
// sources 52.8.
constexpr int kHotWarps = 32;
constexpr int kHotSlots =
    (int)((162 * 1024 - 256 - kHotWarps * sizeof(PrStage)) / sizeof(float) / 1024) * 1024;
constexpr size_t kHotSmem = kHotSlots * sizeof(float) + kHotWarps * sizeof(PrStage);
constexpr int kHotBuckets = 1024;
// In-edges from which on, and the share of them with a hot source from which
// on, the copy is made.  us per run without / with: R-MAT, 4.3 M edges 1680 /
// 1715, 7.9 M 2479 / 2385, 12 M 3269 / 2950; Erdos-Renyi, 9 to 18 M edges, a
// share of 78 % 250 / 262 (the contributions fit L1), 47 % 312 / 297, 29 % 426
// / 407, 20 % 563 / 585, 12 % 549 / 556.
constexpr int kHotMinEdges = 1 << 23;
constexpr double kHotMinShare = 0.25;

struct PrHot {
  uint32_t count[kHotBuckets];  // vertices by out-degree bucket
  uint32_t edges[kHotBuckets];  // and their out-edges
  int32_t bucket;               // hot: buckets from this one on
  int32_t n;                    // hot vertices
  uint32_t covered;             // their out-edges
  int32_t next;                 // slots given out
};

// Out-degree buckets: exact below 64, 32 to an octave above.
__device__ __forceinline__ int hot_bucket(int d) {
  if (d < 64) return d;
  const int l = 31 - __clz(d);
  return 64 + (l - 6) * 32 + ((d >> (l - 5)) & 31);
}

__global__ void __launch_bounds__(kNT) k_hot_count(const int32_t *csr_off, int nV, PrHot *h) {
  __shared__ uint32_t s_n[kHotBuckets], s_e[kHotBuckets];
  for (int i = threadIdx.x; i < kHotBuckets; i += kNT) s_n[i] = s_e[i] = 0u;
  __syncthreads();
  for (int v = blockIdx.x * kNT + threadIdx.x; v < nV; v += gridDim.x * kNT) {
    const int d = csr_off[v + 1] - csr_off[v];
    if (d == 0) continue;
    const int b = hot_bucket(d);
    atomicAdd(&s_n[b], 1u);
    atomicAdd(&s_e[b], (uint32_t)d);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kHotBuckets; i += kNT)
    if (s_n[i]) {
      atomicAdd(&h->count[i], s_n[i]);
      atomicAdd(&h->edges[i], s_e[i]);
    }
}

// The lowest bucket from which on all vertices have a slot.
__global__ void __launch_bounds__(kHotBuckets) k_hot_pick(PrHot *h) {
  __shared__ uint32_t s_n[kHotBuckets], s_e[kHotBuckets];
  s_n[threadIdx.x] = h->count[threadIdx.x];
  s_e[threadIdx.x] = h->edges[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) {
    int b = kHotBuckets;
    uint32_t n = 0, e = 0;
    while (b > 1 && n + s_n[b - 1] <= (uint32_t)kHotSlots) {
      --b;
      n += s_n[b];
      e += s_e[b];
    }
    h->bucket = b;
    h->n = (int32_t)n;
    h->covered = e;
  }
}

__global__ void __launch_bounds__(kNT)
    k_hot_assign(const int32_t *csr_off, int nV, PrHot *h, int32_t *hot_id, int32_t *slot_of) {
  const int bucket = h->bucket;
  for (int v = blockIdx.x * kNT + threadIdx.x; v < nV; v += gridDim.x * kNT) {
    const int d = csr_off[v + 1] - csr_off[v];
    int s = -1;
    if (d > 0 && hot_bucket(d) >= bucket) {
      s = atomicAdd(&h->next, 1);
      hot_id[s] = v;
    }
    slot_of[v] = s;
  }
}

// In-edges with a hot source's slot (complemented) in place of its number.
__global__ void __launch_bounds__(kNT)
    k_hot_sources(const int32_t *__restrict__ csc_src, int nE,
                  const int32_t *__restrict__ slot_of, int32_t *__restrict__ out) {
  const long long stride = (long long)gridDim.x * kNT;
  for (long long i = blockIdx.x * (long long)kNT + threadIdx.x; i < nE; i += 4 * stride) {
    int u[4], s[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = i + k * stride < nE ? __ldg(csc_src + i + k * stride) : 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] = __ldg(slot_of + u[k]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * stride < nE) out[i + k * stride] = s[k] >= 0 ? ~s[k] : u[k];
  }
}

// The hot sources' contributions of this iteration, next to one another.
__global__ void __launch_bounds__(kNT)
    k_hot_values(PrBufs bufs, const int32_t *hot_id, int n, float *hot,
                 const gas_counters *cnt) {
  const float *contrib = bufs.contrib[cnt->iteration & 1];
  const int i = blockIdx.x * kNT + threadIdx.x;
  if (i < n) hot[i] = contrib[hot_id[i]];
}

struct PrCarry {
  int32_t row;   // -1: no record
  int32_t done;  // head: the row ends in this tile
  float s, c;
};

// Rows ended before each tile, and the row-end bits (zero before).
__global__ void __launch_bounds__(kNT)
    k_pr_tiles(const int32_t *ne_end, int n_ne, int n_tiles, int32_t *tile_row,
               uint32_t *end_bits) {
  const int tid = blockIdx.x * kNT + threadIdx.x, nthr = gridDim.x * kNT;
  for (int t = tid; t < n_tiles; t += nthr) {
    const int e0 = t * kPrW;
    int lo = 0, hi = n_ne;
    while (lo < hi) {
      const int m = (lo + hi) >> 1;
      if (ne_end[m] <= e0)
        lo = m + 1;
      else
        hi = m;
    }
    tile_row[t] = lo;
  }
  for (int i = tid; i < n_ne; i += nthr) {
    const int last = ne_end[i] - 1;
    atomicOr(end_bits + (last >> 5), 1u << (last & 31));
  }
}

__device__ __forceinline__ int32_t pr_ld_stream(const int32_t *p) {
  int32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// kHot: pol.csc_src holds slots of hot sources, whose contributions are read
// from the CTA's copy.
template <bool kHot>
__global__ void __launch_bounds__(kHot ? kHotWarps * 32 : kNT, kHot ? 1 : kPrCtas)
    k_pr_gather(PrPol pol, PrBufs bufs, const int32_t *ne_vid, const uint32_t *end_bits, int nE,
                const int32_t *tile_row, int n_tiles, PrCarry *head, PrCarry *tail,
                const float *hot, int n_hot, const gas_counters *cnt, double *l1_part) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kPrWarps = kHot ? kHotWarps : kNT / 32;
  extern __shared__ float4 s_dyn[];
  float *s_hot = reinterpret_cast<float *>(s_dyn);
  pr_bind(pol, bufs, cnt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PrStage &stage = reinterpret_cast<PrStage *>(s_hot + (kHot ? kHotSlots : 0))[warp];
  float *s_val = stage.val;
  float *s_sum = stage.sum;
  const int nwarps = gridDim.x * kPrWarps;
  // software pipeline: the next tile's edge indices, row and row ends load
  // while this tile's gathers and sums run
  int tile = blockIdx.x * kPrWarps + warp;
  int r0 = 0;
  uint32_t word = 0;  // row ends of the tile's edges [32 (lane / 4), + 32)
  bool split = false; // row r0 started in an earlier tile
  int idx[kPrK];
  if (tile < n_tiles) {
    r0 = tile_row[tile];
    word = end_bits[tile * (kPrW / 32) + lane / 4];
    split = tile > 0 && !(end_bits[tile * (kPrW / 32) - 1] >> 31);
#pragma unroll
    for (int k = 0; k < kPrK; ++k) {
      const int j = lane + 32 * k;
      idx[k] = j < nE - tile * kPrW ? pr_ld_stream(pol.csc_src + tile * kPrW + j) : 0;
    }
  }
  if constexpr (kHot) {  // hot has room for a whole number of float4
    const float4 *from = reinterpret_cast<const float4 *>(hot);
#pragma unroll 4
    for (int i = threadIdx.x; i < (n_hot + 3) / 4; i += kHotWarps * 32) s_dyn[i] = from[i];
    __syncthreads();
  }
  for (; tile < n_tiles; tile += nwarps) {
    const int ne = nE - tile * kPrW;
    float val[kPrK];
#pragma unroll
    for (int k = 0; k < kPrK; ++k) {
      const int j = lane + 32 * k;
      val[k] = j < ne && (!kHot || idx[k] >= 0) ? __ldg(pol.contrib + idx[k]) : 0.0f;
    }
    // in registers of their own: a load into val would wait for the first one
    float near[kPrK];
    if constexpr (kHot) {
#pragma unroll
      for (int k = 0; k < kPrK; ++k) near[k] = idx[k] < 0 ? s_hot[~idx[k]] : 0.0f;
    }
    // rows that end before this lane's edges, and in the tile
    const unsigned mine = (word >> (8 * (lane & 3))) & 0xffu;
    int upto = __popc(word);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(FULL, upto, o);
      if (lane >= o) upto += u;
    }
    const int nrows = __shfl_sync(FULL, upto, 31);
    int r = upto - __popc(word >> (8 * (lane & 3)));
    const bool open = !(__shfl_sync(FULL, word, 31) >> 31) && ne > kPrW;
    const int next = tile + nwarps;
    int nr0 = 0;
    uint32_t nword = 0;
    bool nsplit = false;
    if (next < n_tiles) {
      nr0 = tile_row[next];
      nword = end_bits[next * (kPrW / 32) + lane / 4];
      nsplit = !(end_bits[next * (kPrW / 32) - 1] >> 31);
#pragma unroll
      for (int k = 0; k < kPrK; ++k) {
        const int j = lane + 32 * k;
        idx[k] = j < nE - next * kPrW ? pr_ld_stream(pol.csc_src + next * kPrW + j) : 0;
      }
    }
    // the epilogue's inputs for the tile's first 32 rows
    int v0 = 0;
    float inv0 = 0.0f, old0 = 0.0f;
    if (lane < nrows) {
      v0 = __ldg(ne_vid + r0 + lane);
      inv0 = __ldg(pol.inv_deg + v0);
      old0 = pol.rank_old[v0];
    }
#pragma unroll
    for (int k = 0; k < kPrK; ++k) {
      if constexpr (kHot) val[k] = __int_as_float(__float_as_int(val[k]) | __float_as_int(near[k]));
      s_val[pr_pad(lane + 32 * k)] = val[k];
    }
    __syncwarp();
    float acc = 0.0f, first = 0.0f;
    const int first_r = r;
#pragma unroll
    for (int k = 0; k < kPrK; ++k) {
      acc = __fadd_rn(acc, s_val[pr_pad(lane * kPrK + k)]);
      if ((mine >> k) & 1u) {
        if (r == first_r)
          first = acc;
        else
          s_sum[r] = acc;
        acc = 0.0f;
        ++r;
      }
    }
    // segmented inclusive scan of the open-row partials (a lane that ended
    // a row starts a segment)
    const unsigned starts = __ballot_sync(FULL, mine != 0) & (FULL >> (31 - lane));
    const int reach = lane - (starts ? 31 - __clz(starts) : 0);
    PrVal v{acc, 0.0f};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const PrVal u{__shfl_up_sync(FULL, v.s, o), __shfl_up_sync(FULL, v.c, o)};
      if (o <= reach) v = two_sum_add(u, v);
    }
    PrVal cin{__shfl_up_sync(FULL, v.s, 1), __shfl_up_sync(FULL, v.c, 1)};
    if (lane == 0) cin = PrVal{0.0f, 0.0f};
    PrVal row0{0.0f, 0.0f};
    if (mine) {
      row0 = two_sum_add(cin, PrVal{first, 0.0f});
      s_sum[first_r] = __fadd_rn(row0.s, row0.c);
    }
    const PrVal tot{__shfl_sync(FULL, v.s, 31), __shfl_sync(FULL, v.c, 31)};
    __syncwarp();
    // rows that start and end in this tile
    if (lane < nrows && !(lane == 0 && split))
      pol.emit(v0, PrVal{s_sum[lane], 0.0f}, inv0, old0);
    for (int i = lane + 32; i < nrows; i += 32)
      pol.emit(__ldg(ne_vid + r0 + i), PrVal{s_sum[i], 0.0f});
    // the lane that ended the tile's first row has the head record, if that
    // row came from an earlier tile
    if (mine && first_r == 0)
      head[tile] = split ? PrCarry{__ldg(ne_vid + r0), 1, row0.s, row0.c}
                         : PrCarry{-1, 0, 0.0f, 0.0f};
    if (lane == 0) {
      PrCarry tl{-1, 0, 0.0f, 0.0f};
      if (nrows == 0) head[tile] = split ? PrCarry{__ldg(ne_vid + r0), 0, tot.s, tot.c} : tl;
      if (open && !(split && nrows == 0))
        tl = PrCarry{__ldg(ne_vid + r0 + nrows), 0, tot.s, tot.c};
      tail[tile] = tl;
    }
    __syncwarp();
    r0 = nr0;
    word = nword;
    split = nsplit;
  }
  block_sum_store(pol.l1, l1_part + blockIdx.x);
}

// Rows that span tiles.  A thread per tile with a tail record: when the
// next tile's head ends the row (a row of fewer than about kPrW in-edges),
// the two parts are the row.  Longer rows are walked by the whole warp, 32
// head records at a time, up to the tile the row ends in.  A broken chain
// sets the device error word instead of a rank.  And in the first two
// iterations the rows without in-edges, whose ranks (in both buffers) are
// the same ever after.
__global__ void __launch_bounds__(kNT)
    k_pr_join(PrPol pol, PrBufs bufs, const PrCarry *head, const PrCarry *tail, int n_tiles,
              const int32_t *csc_off, int nV, gas_counters *cnt, double *l1_part) {
  pr_bind(pol, bufs, cnt);
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * kNT;
  bool bad = false;
  for (int t0 = blockIdx.x * kNT + (threadIdx.x & ~31); t0 < n_tiles; t0 += stride) {
    const int t = t0 + lane;
    PrCarry tl{-1, 0, 0.0f, 0.0f};
    if (t < n_tiles) tl = tail[t];
    bool walk = false;
    if (tl.row >= 0) {
      if (t + 1 < n_tiles) {
        const PrCarry h = head[t + 1];
        bad |= h.row != tl.row;
        if (h.done)
          pol.emit(tl.row, two_sum_add(PrVal{tl.s, tl.c}, PrVal{h.s, h.c}));
        else
          walk = true;
      } else {
        bad = true;
      }
    }
    unsigned m = __ballot_sync(0xffffffffu, walk);
    while (m) {
      const int src_lane = __ffs(m) - 1;
      m &= m - 1;
      const int wt = __shfl_sync(0xffffffffu, t, src_lane);
      const int row = __shfl_sync(0xffffffffu, tl.row, src_lane);
      PrVal sum{__shfl_sync(0xffffffffu, tl.s, src_lane),
                __shfl_sync(0xffffffffu, tl.c, src_lane)};
      if (lane != 0) sum = PrVal{0.0f, 0.0f};
      bool done = false;
      for (int c = wt + 1; c < n_tiles && !done; c += 32) {
        const int i = c + lane;
        PrCarry h{-1, 0, 0.0f, 0.0f};
        if (i < n_tiles) h = head[i];
        const unsigned dm = __ballot_sync(0xffffffffu, i < n_tiles && h.done);
        const int stop = dm ? __ffs(dm) - 1 : 31;
        if (lane <= stop && i < n_tiles) {
          bad |= h.row != row;
          sum = two_sum_add(sum, PrVal{h.s, h.c});
        }
        done = dm != 0u;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const PrVal u{__shfl_down_sync(0xffffffffu, sum.s, o),
                      __shfl_down_sync(0xffffffffu, sum.c, o)};
        sum = two_sum_add(sum, u);
      }
      if (lane == 0) {
        if (done)
          pol.emit(row, sum);
        else
          bad = true;
      }
    }
  }
  if (cnt->iteration < 2)
    for (int v = blockIdx.x * kNT + threadIdx.x; v < nV; v += stride)
      if (csc_off[v] == csc_off[v + 1]) pol.emit(v, PrVal{0.0f, 0.0f});
  if (bad) atomicExch(&cnt->error, (int32_t)GAS_ERR_DEVICE);
  block_sum_store(pol.l1, l1_part + blockIdx.x);
}

// Deterministic sum of the per-CTA residuals; sets the loop condition.
__global__ void __launch_bounds__(kNT)
    k_pr_finish(const double *l1_part, int n, const double *tol_p,
                gas_counters *cnt, double *residual, cudaGraphConditionalHandle h,
                int in_graph) {
  __shared__ double s[kNT];
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += kNT) v += l1_part[i];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int d = kNT / 2; d > 0; d >>= 1) {
    if (threadIdx.x < d) s[threadIdx.x] += s[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double l1 = s[0];
    const double tol = *tol_p;
    const int max_iter = cnt->max_iter;
    *residual = l1;
    const int it = ++cnt->iteration;
    const bool more = !(l1 <= tol);
    if (more && it >= max_iter) cnt->error = GAS_ERR_ITER_CAP;
    cnt->cond = (more && it < max_iter) ? 1 : 0;
    if (in_graph) cudaGraphSetConditional(h, cnt->cond);
  }
}

// Initial ranks: 1/N, e_seed (seed >= 0), or the caller's vector already
// copied into rank; and the reciprocal out-degrees the iterations scale
// contributions by.
__global__ void k_pr_init(float *rank, float *contrib, float *inv_deg, const int32_t *csr_off,
                          int n, float r0, int have_init, int seed) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += gridDim.x * blockDim.x) {
    const int deg = csr_off[v + 1] - csr_off[v];
    const float inv = deg ? __frcp_rn((float)deg) : 0.0f;
    const float r = have_init ? rank[v] : seed < 0 ? r0 : (v == seed ? 1.0f : 0.0f);
    rank[v] = r;
    inv_deg[v] = inv;
    contrib[v] = __fmul_rn(r, inv);
  }
}

struct PrCtx {
  PrPol pol;
  PrBufs bufs;
  int32_t *tile_row;
  PrCarry *head, *tail;
  int n_tiles;
  int merge_grid;
  int fix_grid;
  int n_hot;  // 0: every contribution is gathered from global memory
  double *residual;
};

gas_status_t pr_body(gas_engine *e, cudaStream_t cs,
                     cudaGraphConditionalHandle h, void *vctx) {
  PrCtx *c = static_cast<PrCtx *>(vctx);
  // algorithmic bytes of one iteration: per edge its source index and the
  // source's contribution; per vertex offsets, old and new rank, new
  // contribution
  gas::prof_begin(e, cs, gas::kProfPagerank, 8LL * e->nE + 16LL * e->nV);
  if (c->n_hot) {
    k_hot_values<<<(c->n_hot + kNT - 1) / kNT, kNT, 0, cs>>>(c->bufs, e->pr_hot_id, c->n_hot,
                                                             e->pr_hot_val, e->cnt);
    k_pr_gather<true><<<c->merge_grid, kHotWarps * 32, kHotSmem, cs>>>(
        c->pol, c->bufs, e->ne_vid, e->pr_end_bits, e->nE, c->tile_row, c->n_tiles, c->head,
        c->tail, e->pr_hot_val, c->n_hot, e->cnt, e->pr_l1);
  } else {
    k_pr_gather<false><<<c->merge_grid, kNT, kNT / 32 * sizeof(PrStage), cs>>>(
        c->pol, c->bufs, e->ne_vid, e->pr_end_bits, e->nE, c->tile_row, c->n_tiles, c->head,
        c->tail, nullptr, 0, e->cnt, e->pr_l1);
  }
  k_pr_join<<<c->fix_grid, kNT, 0, cs>>>(c->pol, c->bufs, c->head, c->tail, c->n_tiles,
                                         e->csc_off, e->nV, e->cnt, e->pr_l1 + c->merge_grid);
  gas::prof_end(e, cs);
  k_pr_finish<<<1, kNT, 0, cs>>>(e->pr_l1, c->merge_grid + c->fix_grid, c->residual + 1,
                                 e->cnt, c->residual, h, e->in_graph ? 1 : 0);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

}  // namespace

extern "C" gas_status_t gas_engine_pagerank_precision(
    gas_engine *e, double damping, double tol, int32_t max_iterations,
    float *ranks, gas_run_stats *stats, void *stream) {
  return gas_engine_pagerank_precision_from(e, damping, tol, max_iterations, nullptr,
                                            ranks, stats, stream);
}

namespace {

// Chooses the hot sources of the graph and rewrites a copy of its in-edges,
// once per graph; *n_hot = 0 where that does not pay or has no memory.
// scratch: nV words.
gas_status_t pr_hot_plan(gas_engine *e, int32_t *scratch, cudaStream_t s, int *n_hot) {
  *n_hot = 0;
  if (e->nE < kHotMinEdges || e->edges_on_host) return GAS_OK;
  if (e->pr_hot_known) {
    *n_hot = e->pr_hot_n;
    return GAS_OK;
  }
  e->pr_hot_mem.free();
  // the copy is a quarter of the free memory at most: other objects may need it
  size_t free_bytes = 0, total = 0;
  CUDA_TRY(cudaMemGetInfo(&free_bytes, &total));
  if ((size_t)e->nE * sizeof(int32_t) > free_bytes / 4 ||
      e->pr_hot_mem.alloc({GROUP_PART(e->pr_hot_ctl, sizeof(PrHot)),
                           GROUP_PART(e->pr_hot_id, kHotSlots * sizeof(int32_t)),
                           GROUP_PART(e->pr_hot_val, kHotSlots * sizeof(float)),
                           GROUP_PART(e->pr_hot_src, (size_t)e->nE * sizeof(int32_t))}) !=
          cudaSuccess) {
    cudaGetLastError();
    e->pr_hot_known = true;
    e->pr_hot_n = 0;
    return GAS_OK;
  }
  PrHot *h = static_cast<PrHot *>(e->pr_hot_ctl);
  const int grid = 4 * e->num_sms;
  CUDA_TRY(cudaMemsetAsync(h, 0, sizeof(PrHot), s));
  k_hot_count<<<grid, kNT, 0, s>>>(e->csr_off, e->nV, h);
  k_hot_pick<<<1, kHotBuckets, 0, s>>>(h);
  int32_t got[3];  // bucket, n, covered
  CUDA_TRY(cudaMemcpyAsync(got, &h->bucket, sizeof(got), cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if ((double)(uint32_t)got[2] >= kHotMinShare * e->nE) {
    k_hot_assign<<<grid, kNT, 0, s>>>(e->csr_off, e->nV, h, e->pr_hot_id, scratch);
    k_hot_sources<<<8 * e->num_sms, kNT, 0, s>>>(e->csc_src, e->nE, scratch, e->pr_hot_src);
    CUDA_TRY(cudaGetLastError());
    *n_hot = e->pr_hot_n = got[1];
  } else {
    e->pr_hot_mem.free();
    e->pr_hot_n = 0;
  }
  e->pr_hot_known = true;
  return GAS_OK;
}

gas_status_t pagerank_run(gas_engine *e, double damping, double tol, int32_t max_iterations,
                          const float *init, int32_t seed, float *ranks, gas_run_stats *stats,
                          void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  if (!(damping > 0.0 && damping < 1.0) || !(tol > 0.0))
    return gas::fail(GAS_ERR_INVALID, "damping must be in (0,1), tol > 0");
  if (max_iterations <= 0) max_iterations = 1000;
  if (stats) *stats = gas_run_stats{};
  const int nV = e->nV;
  if (nV == 0) return GAS_OK;
  if (seed >= nV) return gas::fail(GAS_ERR_INVALID, "seed %d outside [0, %d)", seed, nV);
  PrCtx c;
  c.n_tiles = (int)(((long long)e->nE + kPrW - 1) / kPrW);
  if (!e->pr_tile_row) {  // once per graph
    const size_t T = (size_t)c.n_tiles, words = T * (kPrW / 32), v = (size_t)nV * 4;
    CUDA_TRY(e->pr_mem.alloc(
        {GROUP_PART(e->pr_rank[0], v), GROUP_PART(e->pr_rank[1], v),
         GROUP_PART(e->pr_contrib[0], v), GROUP_PART(e->pr_contrib[1], v),
         GROUP_PART(e->pr_inv_deg, v), GROUP_PART(e->pr_seed, sizeof(int32_t)),
         GROUP_PART(e->pr_l1, sizeof(double) * (kPrPartsPerSm * (size_t)e->num_sms + 2)),
         GROUP_PART(e->pr_tile_row, T * 4), GROUP_PART(e->pr_head, T * sizeof(PrCarry)),
         GROUP_PART(e->pr_tail, T * sizeof(PrCarry)), GROUP_PART(e->pr_end_bits, words * 4)}));
    CUDA_TRY(cudaMemsetAsync(e->pr_end_bits, 0, words * 4, S(stream)));
    k_pr_tiles<<<gas::engine_grid(std::max({c.n_tiles, e->n_ne, 1}), kNT, 8 * e->num_sms), kNT, 0,
                 S(stream)>>>(e->ne_end, e->n_ne, c.n_tiles, e->pr_tile_row, e->pr_end_bits);
  }
  c.tile_row = e->pr_tile_row;
  c.head = static_cast<PrCarry *>(e->pr_head);
  c.tail = static_cast<PrCarry *>(e->pr_tail);
  GAS_TRY(pr_hot_plan(e, reinterpret_cast<int32_t *>(e->pr_contrib[1]), S(stream), &c.n_hot));
  int per_sm = 1;
  if (c.n_hot)
    CUDA_TRY(cudaFuncSetAttribute(k_pr_gather<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kHotSmem));
  else
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pr_gather<false>, kNT,
                                                           kNT / 32 * sizeof(PrStage)));
  // resident CTAs only, and none without a tile
  const int warps = c.n_hot ? kHotWarps : kNT / 32;
  c.merge_grid = std::max(1, std::min(e->num_sms * std::min(std::max(per_sm, 1), kPrCtasMost),
                                      (c.n_tiles + warps - 1) / warps));
  // a thread per tile record, at most 16 CTAs per SM: the records' loads
  // are dependent chains, so they want many threads in flight
  c.fix_grid = (int)std::min<long long>((long long)(kPrPartsPerSm - kPrCtasMost) * e->num_sms,
                                        std::max(1, std::max(c.n_tiles, nV / 4) / kNT + 1));
  const int nparts = c.merge_grid + c.fix_grid;
  c.residual = e->pr_l1 + nparts;
  c.pol.csc_src = c.n_hot ? e->pr_hot_src : e->csc_src;
  c.pol.inv_deg = e->pr_inv_deg;
  c.pol.base = (float)((1.0 - damping) / (double)nV);
  c.pol.base_seed = (float)(1.0 - damping);
  c.pol.damping = (float)damping;
  c.pol.seed_p = e->pr_seed;
  c.pol.seed = -1;
  c.pol.l1 = 0.0;
  c.bufs.rank[0] = e->pr_rank[0];
  c.bufs.rank[1] = e->pr_rank[1];
  c.bufs.contrib[0] = e->pr_contrib[0];
  c.bufs.contrib[1] = e->pr_contrib[1];

  // damping is baked into the captured policy: rebuild when it changes
  if (e->graphs[kGraphPagerank] && e->pr_damping != damping) {
    cudaGraphExecDestroy(e->graphs[kGraphPagerank]);
    e->graphs[kGraphPagerank] = nullptr;
  }
  const bool host_loop = gas::host_loop_for(e);
  if (!host_loop && !e->graphs[kGraphPagerank]) {
    GAS_TRY(gas::build_while_graph(e, pr_body, &c, &e->graphs[kGraphPagerank]));
    e->pr_damping = damping;
  }
  CUDA_TRY(cudaMemcpyAsync(c.residual + 1, &tol, sizeof(double),
                           cudaMemcpyHostToDevice, S(stream)));
  CUDA_TRY(cudaMemcpyAsync(e->pr_seed, &seed, sizeof(int32_t), cudaMemcpyHostToDevice,
                           S(stream)));
  if (init)
    CUDA_TRY(cudaMemcpyAsync(e->pr_rank[0], init, (size_t)nV * 4, cudaMemcpyDefault,
                             S(stream)));
  k_pr_init<<<gas::engine_grid(nV, kNT, 8 * e->num_sms), kNT, 0, S(stream)>>>(
      e->pr_rank[0], e->pr_contrib[0], e->pr_inv_deg, e->csr_off, nV, (float)(1.0 / nV),
      init ? 1 : 0, seed);
  k_reset_loop<<<1, 1, 0, S(stream)>>>(e->cnt, max_iterations);
  cudaError_t ce = cudaGetLastError();
  if (host_loop) {
    if (ce == cudaSuccess) GAS_TRY(gas::run_host_loop(e, pr_body, &c, stream));
  } else if (ce == cudaSuccess) {
    ce = cudaGraphLaunch(e->graphs[kGraphPagerank], S(stream));
  }
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(S(stream));
  if (ce != cudaSuccess)
    return gas::fail(GAS_ERR_CUDA, "pagerank: %s", cudaGetErrorString(ce));
  gas_counters cnt;
  GAS_TRY(gas_engine_read_counters(e, &cnt, stream));
  if (cnt.error && cnt.error != GAS_ERR_ITER_CAP)
    return gas::loop_status(e, cnt, stream);
  if (cnt.error) CUDA_TRY(cudaMemsetAsync(&e->cnt->error, 0, sizeof(int32_t), S(stream)));
  double resid = 0.0;
  CUDA_TRY(cudaMemcpy(&resid, c.residual, sizeof(double), cudaMemcpyDeviceToHost));
  const int final_buf = cnt.iteration & 1;
  if (ranks)
    CUDA_TRY(cudaMemcpyAsync(ranks, e->pr_rank[final_buf], (size_t)nV * 4,
                             cudaMemcpyDefault, S(stream)));
  CUDA_TRY(cudaStreamSynchronize(S(stream)));
  if (stats) {
    stats->iterations = cnt.iteration;
    stats->pull_iters = cnt.iteration;
    stats->kernel_launches = (c.n_hot ? 4 : 3) * cnt.iteration + 3;
    stats->edges_processed = (int64_t)cnt.iteration * e->nE;
    stats->residual = resid;
    stats->graph_launches = host_loop ? 0 : 1;
  }
  if (!(resid <= tol))
    return gas::fail(GAS_ERR_ITER_CAP, "pagerank: residual %.3e after %d iterations",
                     resid, cnt.iteration);
  return GAS_OK;
}

}  // namespace

extern "C" gas_status_t gas_engine_pagerank_precision_from(
    gas_engine *e, double damping, double tol, int32_t max_iterations,
    const float *init, float *ranks, gas_run_stats *stats, void *stream) {
  return pagerank_run(e, damping, tol, max_iterations, init, -1, ranks, stats, stream);
}

extern "C" gas_status_t gas_engine_ppr_precision(gas_engine *e, int32_t seed, double damping,
                                                 double tol, int32_t max_iterations,
                                                 float *ranks, gas_run_stats *stats,
                                                 void *stream) {
  if (seed < 0) return gas::fail(GAS_ERR_INVALID, "ppr: seed must be >= 0");
  return pagerank_run(e, damping, tol, max_iterations, nullptr, seed, ranks, stats, stream);
}
