// gas_sched.h -- fast schedules of the built-in programs (not installed).
#ifndef GAS_SCHED_H_
#define GAS_SCHED_H_

#include <cuda_runtime.h>

#include "gas.h"

struct gas_engine;

namespace gas {

// WHILE(cond) { body } as an instantiated CUDA graph; body captures one
// iteration on the given stream and ends with a kernel that calls
// cudaGraphSetConditional on the handle.
gas_status_t build_while_graph(
    gas_engine *e,
    gas_status_t (*body)(gas_engine *, cudaStream_t, cudaGraphConditionalHandle,
                         void *),
    void *ctx, cudaGraphExec_t *out);

// PUSH / PULL / AUTO schedules of BFS, SSSP, CC (and PageRank falls back to
// the generic kernels): same iteration count and vertex data as run().
gas_status_t run_fast(gas_engine *e, gas_schedule_t schedule,
                      int32_t max_iterations, gas_run_stats *stats,
                      void *stream);

bool host_loop_for(const gas_engine *e);

// What the two one-kernel paths below keep with a graph: bitmaps or the second
// values, the control word, both queues.
struct SmallBytes {
  size_t values, ctl, queues;
  size_t all() const { return values + ctl + queues; }
};
// Up to this many bytes come with set_graph's one allocation: a cudaMalloc of
// their own made the first BFS on R-MAT 2^16 take 242 us (167 us with little
// to allocate).
constexpr size_t kSmallWithGraph = (size_t)16 << 20;
SmallBytes bfs_small_bytes(int64_t nV, int64_t nE);
SmallBytes min_small_bytes(int64_t nV, int64_t nE);

// Launches such a kernel as a cooperative grid with a CTA per kCtaEdges
// vertices and edges; where that is at most cluster_upto CTAs, as one cluster
// of up to kClusterMost.
constexpr int kCtaEdges = 2048;  // 8192 and more: 1.3x and more slower below 100 K edges
constexpr int kClusterMost = 16;
cudaError_t launch_small(void *grid_fn, void *cluster_fn, int cluster_upto, const gas_engine *e,
                         void **args, cudaStream_t s);

// BFS on a graph of at most kBfsSmallMaxV vertices as one cooperative
// kernel (gas_small.cu): same depths and iteration count as run_fast.
// reserve: the kernel's buffers, kept with the graph; false if there is no
// memory for them (the multi-kernel loop needs less).
bool bfs_small_eligible(const gas_engine *e, gas_schedule_t schedule);
bool bfs_small_reserve(gas_engine *e);
gas_status_t run_bfs_small(gas_engine *e, gas_schedule_t schedule, int32_t max_iterations,
                           gas_run_stats *stats, void *stream);

// SSSP and CC from the full active set on a graph of at most kMinSmallMaxV
// vertices as one cooperative kernel (gas_small_min.cu): same vertex data
// and iteration count as run_fast.
bool min_small_eligible(const gas_engine *e, gas_schedule_t schedule);
bool min_small_reserve(gas_engine *e);
gas_status_t run_min_small(gas_engine *e, int32_t max_iterations, gas_run_stats *stats,
                           void *stream);

// The loop of build_while_graph as direct launches (GAS_HOST_LOOP=1).
gas_status_t run_host_loop(
    gas_engine *e,
    gas_status_t (*body)(gas_engine *, cudaStream_t, cudaGraphConditionalHandle,
                         void *),
    void *ctx, void *stream);

// Status of a finished device loop from its counters (clears the error word).
gas_status_t loop_status(gas_engine *e, const gas_counters &c, void *stream);

}  // namespace gas

#endif  // GAS_SCHED_H_
