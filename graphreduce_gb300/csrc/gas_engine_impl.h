// gas_engine_impl.h -- the engine object shared by libgas translation units
// (not installed).
#ifndef GAS_ENGINE_IMPL_H_
#define GAS_ENGINE_IMPL_H_

#include <cuda_runtime.h>

#include <initializer_list>
#include <vector>

#include "gas.h"
#include "gas_internal.h"

#define CUDA_TRY(call)                                                       \
  do {                                                                       \
    cudaError_t e_ = (call);                                                 \
    if (e_ != cudaSuccess)                                                   \
      return gas::fail(GAS_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__,     \
                       #call, cudaGetErrorString(e_));                       \
  } while (0)

#define GAS_TRY(call)                  \
  do {                                 \
    gas_status_t s_ = (call);          \
    if (s_ != GAS_OK) return s_;       \
  } while (0)

// Device arrays that are allocated and freed together, in one cudaMalloc (each
// costs 50 to 200 us, and a first run makes up to a dozen).
struct DeviceGroup {
  struct Part {
    void **p;
    size_t bytes;
  };
  void *base = nullptr;
  std::vector<void **> ptrs;
  cudaError_t alloc(std::initializer_list<Part> parts) {
    free();
    size_t total = 0;
    for (const Part &x : parts) total += round(x.bytes);
    const cudaError_t ce = cudaMalloc(&base, total);
    if (ce != cudaSuccess) {
      base = nullptr;
      cudaGetLastError();  // the caller has it: not for the next launch to report
      return ce;
    }
    size_t at = 0;
    for (const Part &x : parts) {
      *x.p = static_cast<char *>(base) + at;
      ptrs.push_back(x.p);
      at += round(x.bytes);
    }
    return cudaSuccess;
  }
  void free() {
    if (base) cudaFree(base);
    base = nullptr;
    for (void **p : ptrs) *p = nullptr;
    ptrs.clear();
  }
  static size_t round(size_t n) { return (n + 255) / 256 * 256 + (n == 0 ? 256 : 0); }
};
#define GROUP_PART(ptr, bytes) \
  DeviceGroup::Part { reinterpret_cast<void **>(&(ptr)), (size_t)(bytes) }

// ---------------------------------------------------------------------------
// The engine object.
// ---------------------------------------------------------------------------
// BFS runs on graphs up to this many vertices take the one-kernel path
// (figures in gas_small.cu: on every graph measured to this size the faster
// one; at 2^24 it wins on R-MAT and loses on some Erdos-Renyi graphs).
constexpr int kBfsSmallMaxV = 1 << 23;
// ... but with tracing or profiling on, to which the multi-kernel loop gives
// records per iteration, only up to this many.
constexpr int kBfsSmallRecordsMaxV = 1 << 18;
// SSSP and CC from the full active set likewise (figures in
// gas_small_min.cu): under AUTO below 2^22 vertices; the kernel still halves
// the fixed heuristic's time there, but from there on LEARNED's multi-kernel
// push is the faster schedule and the heuristic stays what it is compared
// with.  Under LEARNED up to 2^21 for SSSP (901 against 978 us on R-MAT,
// Erdos-Renyi 2092 against 2367), to 2^20 for CC (at 2^21 824 against 731).
constexpr int kMinSmallMaxV = (1 << 22) - 1;
constexpr int kSsspSmallLearnedMaxV = 1 << 21;
constexpr int kCcSmallLearnedMaxV = 1 << 20;

// Instantiated CUDA graphs cached per engine (valid until the next
// set_graph, since their kernels capture the engine's buffers).
enum { kGraphGeneric = 0, kGraphOrdered = 1, kGraphPagerank = 2, kGraphUser = 3,
       kGraphFast0 = 4, kGraphSlots = 12 };

struct gas_engine {
  gas_program_t prog = GAS_PROG_USER;
  size_t vbytes = 0, gbytes = 0, ebytes = 0;
  int32_t nV = 0, nE = 0;
  void *host_vd = nullptr;
  void *host_ed = nullptr;             // caller's edge data (user engines)
  std::vector<int32_t> h_csr_perm;     // edge-list index of each CSR edge
  std::vector<int32_t> h_csr_to_csc;   // CSC position of each CSR edge
  int32_t *csr_to_csc = nullptr;       // device copy (on first scatter)
  bool edges_dirty = false;            // a user scatter may have changed edge data
  int edge_place = GAS_EDGES_DEVICE;   // placement for the next set_graph
  bool edges_on_host = false;          // csc_src/csr_dst/csc_ed/csr_ed are pinned host memory
  // one allocation for the arrays every graph has, and the pointers into it
  void *arena = nullptr;
  std::vector<void **> arena_ptrs;

  // device graph
  int32_t *csc_off = nullptr, *csc_src = nullptr, *csr_off = nullptr,
          *csr_dst = nullptr;
  void *csc_ed = nullptr, *csr_ed = nullptr;

  // device vertex + frontier state
  void *vd = nullptr;
  int32_t *act = nullptr, *scan = nullptr;
  uint8_t *ret = nullptr;
  void *slot = nullptr, *gres = nullptr;
  uint32_t *bits = nullptr;
  void *xlist = nullptr;       // in-edges past the first of each row, in chunks
  int32_t *xlist_n = nullptr;
  uint32_t *changed = nullptr;  // expansion: vertices whose apply returned true
  void *tile_first = nullptr, *tile_carry = nullptr;
  int32_t *tile_a0 = nullptr;
  int32_t tile_cap = 0;
  int32_t *tpart = nullptr;  // tile partitions of the current frontier pass
  bool tpart_valid = false;  // the compaction wrote them for the active list
  void *xchunks = nullptr, *xctl = nullptr;  // expansion: heavy-row chunks, control word
  void *cpart = nullptr;     // compaction totals (pairs): blocks, then warps
  int32_t n_cblocks = 0;
  gas_counters *cnt = nullptr;
  gas_counters *h_cnt = nullptr;  // pinned

  // precision PageRank buffers (lazily allocated)
  float *pr_rank[2] = {nullptr, nullptr};
  float *pr_contrib[2] = {nullptr, nullptr};
  int32_t *pr_seed = nullptr;  // personalization seed of the run (-1: none)
  float *pr_inv_deg = nullptr;  // [V] RN(1 / out-degree) (0: none)
  double *pr_l1 = nullptr;
  // tiles of the in-edges: rows ended before each, head and tail carry records
  int32_t *pr_tile_row = nullptr;
  void *pr_head = nullptr, *pr_tail = nullptr;
  uint32_t *pr_end_bits = nullptr;  // the last in-edges of the rows
  DeviceGroup pr_mem;
  // hot sources of the graph (gas_runs.cu): their numbers, the iteration's
  // contributions, the in-edges with their slots
  void *pr_hot_ctl = nullptr;
  int32_t *pr_hot_id = nullptr, *pr_hot_src = nullptr;
  float *pr_hot_val = nullptr;
  DeviceGroup pr_hot_mem;
  int32_t pr_hot_n = 0;
  bool pr_hot_known = false;
  double pr_damping = 0.0;

  // fast-schedule state (lazily allocated): frontier queue of C_k with the
  // values its members had at the end of iteration k, out-degree scan,
  // changed bitmap (being built), membership bitmap of C_k, snapshots
  int32_t *q_ids = nullptr, *q_vals = nullptr, *q_end = nullptr, *q_delta = nullptr;
  int32_t *snap = nullptr, *qpart = nullptr;
  uint32_t *cbits = nullptr;
  DeviceGroup fast_mem;  // all of them
  bool graph_only = false;  // holds a batch's union graph: never runs itself
  int32_t pull_div = 4;

  // non-empty in-edge rows of the CSC (dense slab passes)
  int32_t *ne_vid = nullptr, *ne_end = nullptr;
  int32_t n_ne = 0;
  int32_t *ne_scratch = nullptr;
  // warp-slab chunk state: partitions of the dense CSC and of the push
  // queue, per-chunk carries (8-byte values) and fixup rows
  int32_t *slab_dpart = nullptr, *slab_qpart = nullptr, *slab_a0 = nullptr;
  // traces and the learned schedule
  gas_trace_record *trace = nullptr;  // [GAS_TRACE_CAP] device
  int32_t *hist = nullptr;            // [8] degree histogram of the queue
  bool trace_on = false;
  const void *sched_model = nullptr;  // BF16 weights of the schedule head
  int32_t *slab_fix = nullptr;      // chunks needing a fixup, [slab_cap]
  int32_t *slab_fix_n = nullptr;    // their count (reset after each fixup)
  void *slab_first = nullptr, *slab_carry = nullptr;
  int32_t slab_cap = 0;

  // host view of the step API state
  int32_t n_active = 0, n_edges = 0;
  bool counts_dirty = false;
  bool pending_gather = false;
  bool have_gres = false;
  bool slots_pending = false;
  int32_t level = 0;
  int num_sms = 0;
  bool has_graph = false;
  // kernel profiling (gas_engine_set_profiling)
  bool profiling = false;
  cudaEvent_t prof_ev[2] = {nullptr, nullptr};
  int prof_kind = -1;           // kernel bracketed in the current iteration
  int64_t prof_bytes_pending = 0;
  gas_kernel_profile prof = {};
  bool active_full = false;          // active set is [0, nV) from set_active
  bool capturing = false;            // fixed grids (graph capture / host loop)
  bool in_graph = false;             // loop kernels set a graph condition
  cudaGraphExec_t graphs[kGraphSlots] = {};
  bool level_from_counters = false;  // BFS level = counters.iteration
  // small-graph BFS (gas_small.cu): three frontier bitmaps, the control
  // word, the two queues
  uint32_t *sb_bits = nullptr;
  void *sb_ctl = nullptr, *sb_queue = nullptr;
  DeviceGroup sb_mem;
  bool sb_clean = false;  // the kernel left them clear for the next run
  // small-graph SSSP and CC (gas_small_min.cu): second value buffer, the two
  // queues, the control word
  int32_t *sm_vals = nullptr;
  void *sm_queue = nullptr, *sm_ctl = nullptr;
  DeviceGroup sm_mem;
  bool sm_clean = false;
  // what graphs[kGraphUser] was captured with (gas_engine_run_user)
  gas_user_step_fn user_step = nullptr;
  void *user_ctx = nullptr;
  int32_t user_wrote_slots = -1;
};

namespace gas {
// commit pending slots + expansion + compaction of the next frontier, then
// the loop control of a device-side run (the WHILE condition while capturing)
gas_status_t engine_scatter_loop(gas_engine *e, cudaGraphConditionalHandle h, void *stream);
// its kernels
int engine_scatter_kernels(const gas_engine *e);
// one bulk-synchronous iteration of the generic (step API) kernels; the
// frontier's tile partition must be there (engine_partition before the first)
gas_status_t engine_generic_iteration(gas_engine *e, bool ordered,
                                      cudaGraphConditionalHandle h, void *stream);
gas_status_t engine_partition(gas_engine *e, void *stream);
// pieces of it: fused gather+apply into slots / apply only / commit slots
gas_status_t engine_gather_apply(gas_engine *e, void *stream);
gas_status_t engine_apply_only(gas_engine *e, void *stream);
gas_status_t engine_commit(gas_engine *e, void *stream);
// host copy of the counters (synchronises the stream)
gas_status_t engine_sync_counts(gas_engine *e, void *stream);
int engine_grid(int64_t work_items, int per_block, int cap);
// the fast schedule's buffers, with the graph's arrays where a run will want
// them (large BFS, SSSP and CC graphs), so that the first run finds them; not
// where they are more than a quarter of the free memory, as nobody has asked
// for such a run yet
void reserve_fast_buffers(gas_engine *e, void *stream);
bool within_quarter_of_free(size_t bytes);
// CSR/CSC on the device (gas_build.cu): fills csc_off/csc_src/csr_off/
// csr_dst (+ csc_ed/csr_ed), which must be allocated; the permutations
// (edge-list index per CSC / CSR position) when asked for.
gas_status_t build_graph_device(gas_engine *e, const int32_t *srcs, const int32_t *dsts,
                                const void *edge_data, std::vector<int32_t> *csc_perm,
                                std::vector<int32_t> *csr_perm, void *stream);
// Rows of the CSC with in-edges (ne_vid, ne_end; their number to the device
// word n_out); part: ne_blocks(nV) words of scratch.
gas_status_t build_ne_rows(gas_engine *e, int32_t *part, int32_t *n_out, void *stream);
int ne_blocks(int nV);
// Exclusive scan of n device ints in place; part: device_scan_parts(n) ints of
// scratch.
gas_status_t device_scan_excl(int32_t *a, int n, int32_t *part, void *stream);
int device_scan_parts(int n);
// Whether set_graph builds on the device: GAS_GRAPH_BUILD=host|device, else
// from 16,384 edges up.
bool device_build_for(int64_t n_edges);
// grid of a k_partition launch (fixed while capturing)
int engine_partition_grid(gas_engine *e, int64_t items, int tile);
// GAS_HOST_LOOP=1: device loops run as direct launches with one host read
// of the condition per iteration (the kernels are the same; ncu cannot
// profile kernels inside graphs with conditional nodes).
bool host_loop_requested();
// Profiling hooks: bracket one kernel of the current iteration (host loop
// only) and fold its time into the profile once the iteration has run.
enum { kProfPush = 0, kProfPull = 1, kProfPagerank = 2 };
void prof_begin(gas_engine *e, cudaStream_t s, int kind, int64_t bytes);
void prof_end(gas_engine *e, cudaStream_t s);
void prof_collect(gas_engine *e);
}  // namespace gas

#endif  // GAS_ENGINE_IMPL_H_
