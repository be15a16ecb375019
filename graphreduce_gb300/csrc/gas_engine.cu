// gas_engine.cu -- libgas: the GASEngineGPU engine behind the C ABI of
// include/gas.h, for sm_103a.
//
// Layout in HBM per graph (all int32, device resident for the engine's life):
//   csc_off[V+1], csc_src[E], csc_ed[E]    gather side, edge data in CSC order
//   csr_off[V+1], csr_dst[E], csr_ed[E]    scatter side
// Frontier state (V-sized, reused every iteration):
//   active[V] ascending ids, active_scan[V+1] in-degree scan, apply_ret[V],
//   slot[V] new vertex data per active slot, gather_tmp[V], next-frontier
//   bitmap bits[V/32], the expansion's chunk list, per-tile carries.
// Counters live in one device line (gas_counters); the step API reads them
// back once per nextIter()/countActive(), the fast runs never do until the
// end (the loop is a CUDA graph with a device-side WHILE condition).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "gas.h"
#include "gas_device.cuh"
#include "gas_internal.h"
#include "gas_engine_impl.h"
#include "gas_sched.h"

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
namespace gas {
namespace {
thread_local char g_err[512];
}
gas_status_t fail(gas_status_t s, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return s;
}
void clear_error() { g_err[0] = 0; }
const char *g_err_ptr() { return g_err; }
}  // namespace gas

using gasdev::kNT;
using gasdev::SegSource;

// ---------------------------------------------------------------------------
// Built-in vertex programs (device restatements of the reference's four).
// ---------------------------------------------------------------------------
namespace progs {

// sssp.cu:25-66
struct Sssp {
  typedef int32_t VertexData;
  typedef int32_t EdgeData;
  typedef int32_t GatherResult;
  static constexpr int32_t gatherZero = INT_MAX - 100000;
  __device__ static int32_t gatherReduce(const int32_t &a, const int32_t &b) {
    return a < b ? a : b;
  }
  __device__ static int32_t gatherMap(const int32_t *, const int32_t *s,
                                      const int32_t *e) {
    return *s + *e;
  }
  __device__ static bool apply(int32_t *c, const int32_t &d) {
    const bool ch = d < *c;
    if (ch) *c = d;
    return ch;
  }
};

// connected_component.cu:25-63
struct Cc {
  typedef int32_t VertexData;
  typedef int32_t EdgeData;
  typedef int32_t GatherResult;
  static constexpr int32_t gatherZero = INT_MAX;
  __device__ static int32_t gatherReduce(const int32_t &a, const int32_t &b) {
    return a < b ? a : b;
  }
  __device__ static int32_t gatherMap(const int32_t *, const int32_t *s,
                                      const int32_t *) {
    return *s;
  }
  __device__ static bool apply(int32_t *c, const int32_t &l) {
    const bool ch = l < *c;
    if (ch) *c = l;
    return ch;
  }
};

struct PrVertex {
  float rank;
  int32_t numOutEdges;
};

// pagerank.cu:27-73, with explicitly rounded operations so that no FMA
// contraction changes the result relative to the reference's CPU engine.
struct PageRank {
  typedef PrVertex VertexData;
  typedef int32_t EdgeData;
  typedef float GatherResult;
  static constexpr float gatherZero = 0.0f;
  __device__ static float gatherReduce(const float &a, const float &b) {
    return __fadd_rn(a, b);
  }
  __device__ static float gatherMap(const PrVertex *, const PrVertex *s,
                                    const int32_t *) {
    return __fdiv_rn(s->rank, (float)s->numOutEdges);
  }
  __device__ static bool apply(PrVertex *v, const float &g) {
    const float pageConst = 0.15f, tol = 0.01f;
    const float nr = __fadd_rn(pageConst, __fmul_rn(__fsub_rn(1.0f, pageConst), g));
    const bool ret = fabsf(__fsub_rn(nr, v->rank)) >= tol;
    v->rank = nr;
    return ret;
  }
};

}  // namespace progs

// ---------------------------------------------------------------------------
// Program-independent kernels.
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ int warp_incl_sum(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += o;
  }
  return v;
}

// Exclusive prefix sum over the CTA (kNT threads); *total gets the sum.
__device__ __forceinline__ int block_excl_sum(int v, int *total) {
  __shared__ int s_w[kNT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int incl = warp_incl_sum(v);
  if (lane == 31) s_w[warp] = incl;
  __syncthreads();
  int pre = 0, tot = 0;
  for (int w = 0; w < kNT / 32; ++w) {
    if (w < warp) pre += s_w[w];
    tot += s_w[w];
  }
  __syncthreads();
  *total = tot;
  return pre + incl - v;
}

__global__ void k_set_range(int32_t start, int32_t n, const int32_t *csc_off,
                            int32_t *act, int32_t *scan, gas_counters *cnt,
                            int32_t *expand_wait) {
  const int32_t base = csc_off[start];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n;
       i += gridDim.x * blockDim.x) {
    if (i < n) act[i] = start + i;
    scan[i] = csc_off[start + i] - base;
    if (i == n) {
      cnt->n_active = n;
      cnt->n_edges = csc_off[start + n] - base;
      cnt->n_scatter_edges = 0;
      *expand_wait = 0;
    }
  }
}

// vd[act[i]] = slot[i]: makes the applied vertex data visible after every
// gather of the iteration has read the old values (bulk-synchronous apply).
__global__ void k_commit(const int32_t *act, const gas_counters *cnt,
                         const uint8_t *slot, uint8_t *vd, int vbytes) {
  const int n = cnt->n_active;
  if ((vbytes & 3) == 0) {
    const int w = vbytes >> 2;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
      const uint32_t *s = reinterpret_cast<const uint32_t *>(slot) + (size_t)i * w;
      uint32_t *d = reinterpret_cast<uint32_t *>(vd) + (size_t)act[i] * w;
      for (int k = 0; k < w; ++k) d[k] = s[k];
    }
  } else {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
      const uint8_t *s = slot + (size_t)i * vbytes;
      uint8_t *d = vd + (size_t)act[i] * vbytes;
      for (int k = 0; k < vbytes; ++k) d[k] = s[k];
    }
  }
}

// Expansion: set the next-frontier bit of every out-neighbour of every
// apply()==true vertex.  The bit is tested before the atomic: a hub is the
// out-neighbour of many active vertices, and on PageRank (200 K vertices,
// 3 M edges, most of them active) nearly every edge finds its bit set; a
// stale clear bit (plain, L1-cached load) only repeats the same OR.  (A
// second test in L2 before the atomic measured 23 + 22 us for light rows and
// chunks against 19 + 18: the reduction is not waited for, the load is.)
__device__ __forceinline__ void activate(uint32_t *bits, uint32_t w) {
  uint32_t *p = bits + (w >> 5);
  const uint32_t m = 1u << (w & 31);
  if (!(*p & m)) atomicOr(p, m);
}

// Rows of more than kXLight out-edges leave their edges as chunks of kXChunk
// for expand_chunks: at most E / kXLight entries.
constexpr int kXLight = 64;
constexpr int kXChunk = 256;

// k_expand_mark's results: chunks listed, out-edges of the applied vertices.
struct ExpandCtl {
  int32_t n_chunks, n_edges;
  uint32_t missed;  // in-edges a pull looked at in vain
  int32_t wait;     // iterations to push after a pull that missed much
};

// Whether the iteration may pull at all: not if the active vertices have few
// in-edges, so that few out-edges are to be expected of those among them that
// apply, nor just after a bad pull.  (Marking costs an iteration that then
// pushes 2 to 3 us.  1/4, 1/8 and 1/16 of the edges within 1 % of one another.)
constexpr int kXActiveDiv = 8;
__device__ __forceinline__ bool expand_may_pull(const gas_counters *cnt, const ExpandCtl *ctl,
                                                const int2 *list, int nE) {
  return list && ctl->wait == 0 && (long long)cnt->n_edges * kXActiveDiv > nE;
}

// The light rows among a warp's 32 (off, deg), pushed: their edges laid end to
// end, 64 per round.
__device__ __forceinline__ void expand_light(int off, int deg, const int32_t *csr_dst,
                                             uint32_t *bits, int *s_start, int *s_excl) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // without the empty ones, to consecutive places
  const bool light = deg > 0 && deg <= kXLight;
  const unsigned lb = __ballot_sync(FULL, light);
  if (!lb) return;  // warp-uniform
  const int rows = __popc(lb);
  const int incl = warp_incl_sum(light ? deg : 0);
  const int T = __shfl_sync(FULL, incl, 31);
  if (light) {
    const int k = __popc(lb & ((1u << lane) - 1u));
    s_excl[k] = incl - deg;
    s_start[k] = off;
  }
  __syncwarp();
  const bool ok = lane < rows;
  const int excl = ok ? s_excl[lane] : 0;
  const int shift = ok ? s_start[lane] - excl : 0;
  __syncwarp();
  for (int r = 0; r < T; r += 64) {
    int w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r0 = r + 32 * h;
      // the row of edge r0 is the last one starting at or before it; a bit
      // per row that starts inside the round gives the other lanes theirs
      const int row0 = __popc(__ballot_sync(FULL, ok && excl <= r0)) - 1;
      const int k = excl - r0;
      const unsigned starts = __reduce_or_sync(FULL, (ok && k >= 1 && k < 32) ? (1u << k) : 0u);
      int row = row0 + __popc(starts & ((2u << lane) - 1u));
      row = row > 31 ? 31 : row;
      const int pos = r0 + lane + __shfl_sync(FULL, shift, row);
      w[h] = r0 + lane < T ? __ldg(csr_dst + pos) : -1;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (w[h] >= 0) activate(bits, (uint32_t)w[h]);
  }
}

// First pass over the active slots, a warp 32 of them: commits their new
// vertex data (slot != null; vd[act[i]] = slot[i], after every gather of the
// iteration has read the old values), adds up the applied ones' out-edges and
// lists the chunks of their heavy rows (one atomic per warp).  Where a pull
// may follow it marks them in a bitmap, and k_expand chooses the direction;
// elsewhere it pushes the light rows at once.
__global__ void __launch_bounds__(kNT)
    k_expand_mark(const int32_t *act, const gas_counters *cnt, const uint8_t *ret,
                  const int32_t *csr_off, const int32_t *csr_dst, uint32_t *changed,
                  uint32_t *bits, const uint8_t *slot, uint8_t *vd, int vbytes, int2 *chunks,
                  const int2 *list, int nE, ExpandCtl *ctl) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ int s_start[kNT / 32][32], s_excl[kNT / 32][32];
  const bool mark = expand_may_pull(cnt, ctl, list, nE);
  const int n = cnt->n_active;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  int edges = 0;
  for (long long base = 32LL * gwarp; base < n; base += 32LL * nwarps) {
    const long long i = base + lane;
    int off = 0, deg = 0, word = -1;
    uint32_t bit = 0;
    if (i < n) {
      const int v = act[i];
      if (slot) {
        if ((vbytes & 3) == 0) {
          const int w = vbytes >> 2;
          const uint32_t *s = reinterpret_cast<const uint32_t *>(slot) + (size_t)i * w;
          uint32_t *d = reinterpret_cast<uint32_t *>(vd) + (size_t)v * w;
          for (int k = 0; k < w; ++k) d[k] = s[k];
        } else {
          for (int k = 0; k < vbytes; ++k)
            vd[(size_t)v * vbytes + k] = slot[(size_t)i * vbytes + k];
        }
      }
      if (ret[i]) {
        off = csr_off[v];
        deg = csr_off[v + 1] - off;
        word = v >> 5;
        bit = 1u << (v & 31);
      }
    }
    edges += deg;
    // the ids ascend, so a warp's bits are in few words: one reduction each
    if (mark) {  // uniform
      const unsigned same = __match_any_sync(FULL, word);
      const uint32_t all = __reduce_or_sync(same, bit);
      if (word >= 0 && lane == __ffs(same) - 1) atomicOr(changed + word, all);
    }
    unsigned hb = __ballot_sync(FULL, deg > kXLight);
    if (hb) {  // warp-uniform
      const int nc = deg > kXLight ? (deg + kXChunk - 1) / kXChunk : 0;
      const int incl = warp_incl_sum(nc);
      int at = 0;
      if (lane == 31) at = atomicAdd(&ctl->n_chunks, incl);
      at = __shfl_sync(FULL, at, 31) + incl - nc;
      for (; hb; hb &= hb - 1) {
        const int l = __ffs(hb) - 1;
        const int o = __shfl_sync(FULL, off, l), d = __shfl_sync(FULL, deg, l);
        const int p = __shfl_sync(FULL, at, l), c = __shfl_sync(FULL, nc, l);
        for (int k = lane; k < c; k += 32)
          chunks[p + k] = make_int2(o + k * kXChunk, o + min(d, (k + 1) * kXChunk));
      }
    }
    if (!mark) expand_light(off, deg, csr_dst, bits, s_start[warp], s_excl[warp]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) edges += __shfl_xor_sync(FULL, edges, d);
  if (lane == 0 && edges) atomicAdd(&ctl->n_edges, edges);
}

// The heavy rows' chunks, pushed: a warp each, all of a chunk's loads in
// flight.
__device__ __forceinline__ void expand_chunks(const int2 *chunks, int n, const int32_t *csr_dst,
                                              uint32_t *bits) {
  const int lane = threadIdx.x & 31;
  const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int c = gwarp; c < n; c += nwarps) {
    const int2 r = chunks[c];
    int w[kXChunk / 32];
#pragma unroll
    for (int k = 0; k < kXChunk / 32; ++k) {
      const int pos = r.x + 32 * k + lane;
      w[k] = pos < r.y ? __ldg(csr_dst + pos) : -1;
    }
#pragma unroll
    for (int k = 0; k < kXChunk / 32; ++k)
      if (w[k] >= 0) activate(bits, (uint32_t)w[k]);
  }
}

// Pulled: a warp per word of the next frontier, a lane per vertex, which
// looks for a marked in-neighbour among its first kXLight in-edges -- the
// first alone, then four at a time -- and stops at the first.  The in-edges
// after those are chunks of kXChunk, listed once per graph (k_expand_list), a
// warp each, skipped where the vertex has its bit already: hubs that no
// marked vertex leads to would leave whole rows to single warps (CC on R-MAT
// 2^14 with grid islands 2.2 -> 4.3 ms).
__device__ __forceinline__ void expand_pull(const int32_t *csc_off, const int32_t *csc_src,
                                            const uint32_t *changed, int nV, const int2 *list,
                                            int n_list, uint32_t *bits, uint32_t *missed) {
  uint32_t vain = 0;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int w = gwarp; 32LL * w < nV; w += nwarps) {
    const int v = 32 * w + lane;
    // unsigned: the steps past the last edge must not wrap
    uint32_t i = 0, stop = 0;
    if (v < nV) {
      i = csc_off[v];
      stop = min((uint32_t)csc_off[v + 1], i + kXLight);
    }
    const uint32_t look = stop - i;
    bool hit = false;
    if (i < stop) {
      const int u = __ldg(csc_src + i);
      hit = (changed[u >> 5] >> (u & 31)) & 1u;
    }
    for (++i; i < stop && !hit; i += 4) {
      int u[4];
      uint32_t f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = i + j < stop ? __ldg(csc_src + i + j) : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = u[j] >= 0 ? changed[u[j] >> 5] : 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) hit |= u[j] >= 0 && ((f[j] >> (u[j] & 31)) & 1u);
    }
    if (!hit) vain += look;
    const unsigned word = __ballot_sync(FULL, hit);
    if (lane == 0 && word) atomicOr(bits + w, word);
  }
  for (int c = gwarp; c < n_list; c += nwarps) {
    const int2 e = list[c];  // vertex, first in-edge
    uint32_t *p = bits + (e.x >> 5);
    const uint32_t m = 1u << (e.x & 31);
    // the votes below need the whole warp, and other warps set bits of the
    // word meanwhile: the lanes agree on what they have read
    if (__any_sync(FULL, (__ldcg(p) & m) != 0u)) continue;
    const uint32_t end = csc_off[e.x + 1];
    int u[kXChunk / 32];
    bool f = false;
#pragma unroll
    for (int k = 0; k < kXChunk / 32; ++k) {
      const uint32_t q = (uint32_t)e.y + 32 * k + lane;
      u[k] = q < end ? __ldg(csc_src + q) : -1;
    }
#pragma unroll
    for (int k = 0; k < kXChunk / 32; ++k)
      f |= u[k] >= 0 && ((changed[u[k] >> 5] >> (u[k] & 31)) & 1u);
    if (!__any_sync(FULL, f))
      vain += kXChunk / 32;
    else if (lane == 0)
      atomicOr(p, m);
  }
  vain = __reduce_add_sync(FULL, vain);
  if (lane == 0 && vain) atomicAdd(missed, vain);
}

// The in-edges after the first kXLight of each row, in chunks: at most
// E / kXLight entries.
__global__ void __launch_bounds__(kNT)
    k_expand_list(const int32_t *csc_off, int nV, int2 *list, int32_t *n) {
  for (int v = blockIdx.x * kNT + threadIdx.x; v < nV; v += gridDim.x * kNT) {
    const int off = csc_off[v], rest = csc_off[v + 1] - off - kXLight;
    if (rest <= 0) continue;
    const int nc = (rest + kXChunk - 1) / kXChunk;
    const int at = atomicAdd(n, nc);
    for (int k = 0; k < nc; ++k) list[at + k] = make_int2(v, off + kXLight + k * kXChunk);
  }
}

// Sets the next-frontier bit of every out-neighbour of a marked vertex: by
// push, or by pull where the marked vertices have more than 1 / kXPullDiv of
// the edges: a push is bound by the reductions on words that several SMs fill
// at once, a pull has one per word and reads a few in-edges per vertex.  A
// pull that looked at more than 1 / kXMissDiv of the in-edges in vain makes
// the next kXWait iterations push.  us per run, push only (rows and chunks in
// a kernel each) / with 1/2, 1/4, 1/8, 1/16: the reference's PageRank on
// R-MAT 200 K, 3 M edges 3712 / 3010, 2933, 2901, 2900; 20 K 1797 / 1478,
// 1431, 1420, 1448; Erdos-Renyi 200 K 1785 / 1371, 1349, 1331, 1369; run()
// on R-MAT 2^18, CC 418 / 391, 374, 373, -, BFS 217 / 193, 173, 171, -; SSSP on
// R-MAT 2^21 4309 / 4088, 4078, 4091, 4166.  CC on R-MAT 2^14 with 200 grid
// islands, whose pulls would miss: 2147 / 2252, 2271, 2293, and 2200 with the
// rule on misses.
constexpr int kXPullDiv = 8;
constexpr int kXMissDiv = 4;
constexpr int kXWait = 16;
__global__ void __launch_bounds__(kNT)
    k_expand(const int32_t *act, const gas_counters *cnt, const uint8_t *ret,
             const int32_t *csr_off, const int32_t *csr_dst, const int32_t *csc_off,
             const int32_t *csc_src, int nV, int nE, const uint32_t *changed, const int2 *chunks,
             ExpandCtl *ctl, const int2 *list, const int32_t *n_list, uint32_t *bits) {
  __shared__ int s_start[kNT / 32][32], s_excl[kNT / 32][32];
  const bool marked = expand_may_pull(cnt, ctl, list, nE);
  if (marked && (long long)ctl->n_edges * kXPullDiv > nE) {
    expand_pull(csc_off, csc_src, changed, nV, list, *n_list, bits, &ctl->missed);
    return;
  }
  if (marked) {  // the light rows are still to be pushed
    const int n = cnt->n_active, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
    for (long long base = 32LL * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); base < n;
         base += 32LL * nwarps) {
      const long long i = base + lane;
      int off = 0, deg = 0;
      if (i < n && ret[i]) {
        const int v = act[i];
        off = csr_off[v];
        deg = csr_off[v + 1] - off;
      }
      expand_light(off, deg, csr_dst, bits, s_start[warp], s_excl[warp]);
    }
  }
  expand_chunks(chunks, ctl->n_chunks, csr_dst, bits);
}

// Compaction of the next-frontier bitmap into the ascending active list with
// its in-degree scan (scatter_if_mgpu.h:130-157 + the gather's degree scan),
// clearing the bitmap for the following iteration.  A warp owns a run of 16
// words and walks it in two rounds of 8, lane l taking vertex 32 w + l of
// each word: the in-degree loads of a word are coalesced and a round's are
// in flight together.  (A thread per 4 words, the bits of each in a serial
// loop, left 200 K vertices to 7 CTAs: 40 us to count and 91 us to write,
// against 5.4 and 11.)
constexpr int kCWords = 16;                      // words per warp
constexpr int kCRound = 8;
constexpr int kCWarps = kNT / 32;
constexpr int kCBlockWords = kCWords * kCWarps;  // 128 words per block
// Up to this many blocks (8 M vertices) every block of the write pass sums
// the totals before it; beyond, a spine kernel scans them.
constexpr int kCSumBlocks = 2048;

struct CRound {
  int deg[kCRound];
  uint32_t word[kCRound];
};

__device__ __forceinline__ void c_round_load(uint32_t myword, const int32_t *csc_off, int w0,
                                             int r, CRound &q) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kCRound; ++i) {
    q.word[i] = __shfl_sync(0xffffffffu, myword, r + i);
    q.deg[i] = 0;
    if ((q.word[i] >> lane) & 1u) {
      const int v = (w0 + r + i) * 32 + lane;
      q.deg[i] = csc_off[v + 1] - csc_off[v];
    }
  }
}

// Members and in-edges per block (part) and per warp (wpart); also takes
// the expansion's out-edge count and clears its control word and marks.
__global__ void __launch_bounds__(kNT)
    k_compact_count(const uint32_t *bits, uint32_t *changed, const int32_t *csc_off, int nW, int nE,
                    int2 *part, int2 *wpart, ExpandCtl *ctl, gas_counters *cnt) {
  __shared__ int2 s_t[kCWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * kCWarps + warp) * kCWords;
  const uint32_t myword = lane < kCWords && w0 + lane < nW ? bits[w0 + lane] : 0u;
  if (lane < kCWords && w0 + lane < nW) changed[w0 + lane] = 0u;
  const unsigned nz = __ballot_sync(0xffffffffu, myword != 0u);
  int c = __popc(myword), d = 0;
#pragma unroll 1
  for (int r = 0; r < kCWords; r += kCRound) {
    if (!((nz >> r) & ((1u << kCRound) - 1u))) continue;  // warp-uniform
    CRound q;
    c_round_load(myword, csc_off, w0, r, q);
#pragma unroll
    for (int i = 0; i < kCRound; ++i) d += q.deg[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c += __shfl_xor_sync(0xffffffffu, c, o);
    d += __shfl_xor_sync(0xffffffffu, d, o);
  }
  if (lane == 0) {
    s_t[warp] = make_int2(c, d);
    wpart[blockIdx.x * kCWarps + warp] = make_int2(c, d);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int2 t = make_int2(0, 0);
    for (int k = 0; k < kCWarps; ++k) {
      t.x += s_t[k].x;
      t.y += s_t[k].y;
    }
    part[blockIdx.x] = t;
    if (blockIdx.x == 0) {
      cnt->n_scatter_edges = ctl->n_edges;
      ctl->n_edges = 0;
      ctl->n_chunks = 0;
      ctl->wait = (long long)ctl->missed * kXMissDiv > nE ? kXWait : max(ctl->wait - 1, 0);
      ctl->missed = 0;
    }
  }
}

// More than kCSumBlocks blocks: part[] becomes its exclusive scan.
__global__ void __launch_bounds__(kNT) k_compact_spine(int2 *part, int nb) {
  int2 carry = make_int2(0, 0);
  for (int base = 0; base < nb; base += kNT) {
    const int i = base + threadIdx.x;
    const int2 v = i < nb ? part[i] : make_int2(0, 0);
    int tc, td;
    const int ec = block_excl_sum(v.x, &tc);
    const int ed = block_excl_sum(v.y, &td);
    if (i < nb) part[i] = make_int2(carry.x + ec, carry.y + ed);
    carry.x += tc;
    carry.y += td;
  }
}

// Loop control of a device-side run, done by the last block of the
// compaction: one more iteration while the frontier is non-empty and the cap
// is not reached; reaching the cap with work left raises the error word.
struct LoopEnd {
  int on;        // 0: the step API, whose host decides
  int in_graph;  // the condition of a WHILE node is set as well
  cudaGraphConditionalHandle h;
};

// The active list, its in-degree scan and the totals.  tile > 0: also the
// next gather's tile partition -- the merge-path boundary of tile t lies in
// the segment a with a + scan[a] <= t * tile <= a + scan[a + 1], so each
// member writes the boundaries inside its own range and no tile has to
// search for its own (k_partition, 10 us of dependent loads per iteration).
__global__ void __launch_bounds__(kNT)
    k_compact_write(uint32_t *bits, const int32_t *csc_off, int nW, const int2 *part,
                    const int2 *wpart, int scanned, int32_t *act, int32_t *scan,
                    int32_t *tile_part, int tile, gas_counters *cnt, LoopEnd end) {
  constexpr unsigned FULL = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * kCWarps + warp) * kCWords;
  const uint32_t myword = lane < kCWords && w0 + lane < nW ? bits[w0 + lane] : 0u;
  const bool last_block = blockIdx.x == gridDim.x - 1;
  if (!__syncthreads_or(myword != 0u) && !last_block) return;
  int2 base;
  if (scanned) {
    base = part[blockIdx.x];
  } else {
    int c = 0, d = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kNT) {
      const int2 t = part[b];
      c += t.x;
      d += t.y;
    }
    block_excl_sum(c, &base.x);
    block_excl_sum(d, &base.y);
  }
  for (int k = 0; k < warp; ++k) {
    const int2 t = wpart[blockIdx.x * kCWarps + k];
    base.x += t.x;
    base.y += t.y;
  }
  int bq = base.x, bd = base.y;
  const unsigned nz = __ballot_sync(FULL, myword != 0u);
  const unsigned below = (1u << lane) - 1u;
#pragma unroll 1
  for (int r = 0; r < kCWords; r += kCRound) {
    if (!((nz >> r) & ((1u << kCRound) - 1u))) continue;  // warp-uniform
    CRound q;
    c_round_load(myword, csc_off, w0, r, q);
#pragma unroll
    for (int i = 0; i < kCRound; ++i) {
      const uint32_t word = q.word[i];
      if (!word) continue;  // warp-uniform
      const int deg = q.deg[i];
      const int incl = warp_incl_sum(deg);
      const int pos = bq + __popc(word & below), beg = bd + incl - deg;
      int t0 = 0, t1 = -1;
      if ((word >> lane) & 1u) {
        act[pos] = (w0 + r + i) * 32 + lane;
        scan[pos] = beg;
        if (tile) {
          t0 = (int)(((unsigned)(pos + beg) + tile - 1u) / (unsigned)tile);
          t1 = (int)((unsigned)(pos + beg + deg) / (unsigned)tile);
        }
      }
      if (tile) {
        unsigned big = __ballot_sync(FULL, t1 - t0 >= 4);  // hubs, by the whole warp
        if (t1 - t0 < 4)
          for (int t = t0; t <= t1; ++t) tile_part[t] = pos;
        for (; big; big &= big - 1) {
          const int l = __ffs(big) - 1;
          const int p = __shfl_sync(FULL, pos, l), e = __shfl_sync(FULL, t1, l);
          for (int t = __shfl_sync(FULL, t0, l) + lane; t <= e; t += 32) tile_part[t] = p;
        }
      }
      bq += __popc(word);
      bd += __shfl_sync(FULL, incl, 31);
    }
  }
  if (myword) bits[w0 + lane] = 0u;
  if (last_block && warp == kCWarps - 1 && lane == 0) {  // bq, bd: the totals
    scan[bq] = bd;
    cnt->n_active = bq;
    cnt->n_edges = bd;
    // every tile boundary past the last one is the end of the path
    if (tile) tile_part[(int)(((long long)bq + bd + tile - 1) / tile)] = bq;
    if (end.on) {
      const int it = ++cnt->iteration;
      if (bq > 0 && it >= cnt->max_iter) cnt->error = GAS_ERR_ITER_CAP;
      cnt->cond = (bq > 0 && it < cnt->max_iter) ? 1 : 0;
      if (end.in_graph) cudaGraphSetConditional(end.h, cnt->cond);
    }
  }
}

// BFS apply without gather (bfs.cu:58-71): level from the engine.
__global__ void k_bfs_apply(const int32_t *act, const gas_counters *cnt,
                            int32_t *depth, uint8_t *ret, int32_t level,
                            int32_t level_from_counters) {
  const int n = cnt->n_active;
  if (level_from_counters) level = cnt->iteration;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * blockDim.x) {
    int32_t *d = depth + act[i];
    const bool r = *d == -1;
    if (r) *d = level;
    ret[i] = r ? 1 : 0;
  }
}

}  // namespace

namespace {

template <class T>
gas_status_t dalloc(T **p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  cudaError_t e = cudaMalloc((void **)p, n * sizeof(T));
  if (e != cudaSuccess) {
    *p = nullptr;
    return gas::fail(GAS_ERR_NOMEM, "cudaMalloc of %zu bytes: %s",
                     n * sizeof(T), cudaGetErrorString(e));
  }
  return GAS_OK;
}

template <class T>
void dfree(T *&p) {
  if (p) cudaFree((void *)p);
  p = nullptr;
}

// Edge arrays in pinned, mapped host memory (GAS_EDGES_HOST): kernels read
// them over NVLink-C2C through their device address.
template <class T>
gas_status_t halloc(T **p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  void *h = nullptr;
  cudaError_t e = cudaHostAlloc(&h, n * sizeof(T), cudaHostAllocMapped);
  void *d = nullptr;
  if (e == cudaSuccess) e = cudaHostGetDevicePointer(&d, h, 0);
  if (e != cudaSuccess) {
    if (h) cudaFreeHost(h);
    return gas::fail(GAS_ERR_NOMEM, "cudaHostAlloc of %zu bytes: %s", n * sizeof(T),
                     cudaGetErrorString(e));
  }
  if (d != h) {  // kernels and the host must see one address (UVA)
    cudaFreeHost(h);
    return gas::fail(GAS_ERR_UNSUPPORTED, "host edge arrays need unified addressing");
  }
  *p = static_cast<T *>(h);
  return GAS_OK;
}

template <class T>
void hfree(T *&p) {
  if (p) cudaFreeHost((void *)p);
  p = nullptr;
}

// The arrays of set_graph, gathered and then allocated together: some thirty
// cudaMallocs and as many frees took 5 ms of a set_graph of 31 M edges.
struct ArenaPlan {
  gas_engine *e;
  std::vector<size_t> at;
  size_t bytes = 0;
  explicit ArenaPlan(gas_engine *eng) : e(eng) {}
  template <class T>
  void add(T **p, size_t n) {
    *p = nullptr;
    at.push_back(bytes);
    e->arena_ptrs.push_back(reinterpret_cast<void **>(p));
    bytes += (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~(size_t)255;
  }
  gas_status_t alloc() {
    const cudaError_t ce = cudaMalloc(&e->arena, bytes);
    if (ce != cudaSuccess) {
      e->arena = nullptr;
      e->arena_ptrs.clear();
      cudaGetLastError();
      return gas::fail(GAS_ERR_NOMEM, "cudaMalloc of %zu bytes: %s", bytes,
                       cudaGetErrorString(ce));
    }
    for (size_t i = 0; i < at.size(); ++i)
      *e->arena_ptrs[i] = static_cast<uint8_t *>(e->arena) + at[i];
    return GAS_OK;
  }
};

void free_graph(gas_engine *e) {
  if (e->edges_on_host) {
    hfree(e->csc_src); hfree(e->csr_dst); hfree(e->csc_ed); hfree(e->csr_ed);
  }
  e->edges_on_host = false;
  for (void **p : e->arena_ptrs) *p = nullptr;
  e->arena_ptrs.clear();
  dfree(e->arena);
  dfree(e->csr_to_csc);
  e->pr_mem.free();
  e->pr_hot_mem.free();
  e->pr_hot_n = 0;
  e->pr_hot_known = false;
  e->sb_mem.free();
  e->sm_mem.free();
  e->sb_clean = e->sm_clean = false;
  e->h_csr_perm.clear();
  e->h_csr_to_csc.clear();
  e->host_ed = nullptr;
  e->edges_dirty = false;
  e->fast_mem.free();
  e->n_ne = e->slab_cap = 0;
  for (int i = 0; i < kGraphSlots; ++i) {
    if (e->graphs[i]) cudaGraphExecDestroy(e->graphs[i]);
    e->graphs[i] = nullptr;
  }
  e->has_graph = false;
}

size_t program_vbytes(gas_program_t p) {
  switch (p) {
    case GAS_PROG_BFS: case GAS_PROG_SSSP: case GAS_PROG_CC: return 4;
    case GAS_PROG_PAGERANK: return 8;
    default: return 0;
  }
}

inline cudaStream_t S(void *s) { return (cudaStream_t)s; }

int grid_for(int64_t work_items, int per_block, int cap) {
  int64_t g = (work_items + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

template <class K>
int occupancy_grid(gas_engine *e, K kernel, size_t smem = 0) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kNT, smem);
  if (per_sm < 1) per_sm = 1;
  return e->num_sms * per_sm;
}

gas_status_t sync_counts(gas_engine *e, void *stream) {
  CUDA_TRY(cudaMemcpyAsync(e->h_cnt, e->cnt, sizeof(gas_counters),
                           cudaMemcpyDeviceToHost, S(stream)));
  CUDA_TRY(cudaStreamSynchronize(S(stream)));
  e->n_active = e->h_cnt->n_active;
  e->n_edges = e->h_cnt->n_edges;
  e->counts_dirty = false;
  return GAS_OK;
}

// Merge items per gather tile of the built-in programs (4-byte values).
constexpr int kBuiltinTile = gasdev::TileShape<4>::kTile;

// Launch the generic gather (fused with apply or not) for program P;
// partitioned: the compaction that made the frontier wrote its partition.
template <class P>
gas_status_t launch_generic_gather(gas_engine *e, bool fuse, bool ordered,
                                   bool partitioned, void *stream) {
  using GR = typename P::GatherResult;
  gasdev::GenericGather<P> pol;
  pol.csc_src = e->csc_src;
  pol.csc_ed = static_cast<const typename P::EdgeData *>(e->csc_ed);
  pol.vd = static_cast<const typename P::VertexData *>(e->vd);
  pol.slot = static_cast<typename P::VertexData *>(e->slot);
  pol.ret = e->ret;
  pol.gres = static_cast<GR *>(e->gres);
  pol.fuse = fuse ? 1 : 0;
  if (ordered) {
    const int g = e->capturing ? 8 * e->num_sms : grid_for(e->n_active, kNT, 65535);
    gasdev::k_gather_ordered<P><<<g, kNT, 0, S(stream)>>>(pol, e->act,
                                                          e->csc_off, e->cnt);
    CUDA_TRY(cudaGetLastError());
    return GAS_OK;
  }
  const SegSource src = gasdev::frontier_source(
      e->act, e->scan, e->csc_off, &e->cnt->n_active, &e->cnt->n_edges, e->tpart);
  constexpr int kTile = gasdev::TileShape<sizeof(GR)>::kTile;
  static_assert(kTile == kBuiltinTile, "the compaction writes this tile's partition");
  const int64_t items = (int64_t)e->n_active + e->n_edges;
  if (!partitioned)
    gasdev::k_partition<kTile, false>
        <<<gas::engine_partition_grid(e, items, kTile), 256, 0, S(stream)>>>(src, e->tpart);
  const int cap = occupancy_grid(e, gasdev::k_gather_tiles<P>);
  const int grid = e->capturing ? cap : grid_for(items, kTile, cap);
  gasdev::k_gather_tiles<P><<<grid, kNT, 0, S(stream)>>>(
      pol, src, static_cast<GR *>(e->tile_first),
      static_cast<GR *>(e->tile_carry), e->tile_a0);
  CUDA_TRY(cudaGetLastError());
  const int64_t ntiles = (items + kTile - 1) / kTile;
  const int fgrid = e->capturing ? 4 * e->num_sms
                                  : grid_for(ntiles, kNT / 32, 4 * e->num_sms);
  gasdev::k_gather_fixup<P><<<fgrid, kNT, 0, S(stream)>>>(
      pol, src, static_cast<GR *>(e->tile_first),
      static_cast<GR *>(e->tile_carry), e->tile_a0);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

gas_status_t builtin_gather(gas_engine *e, bool fuse, bool ordered,
                            bool partitioned, void *stream) {
  switch (e->prog) {
    case GAS_PROG_SSSP:
      return launch_generic_gather<progs::Sssp>(e, fuse, ordered, partitioned, stream);
    case GAS_PROG_CC:
      return launch_generic_gather<progs::Cc>(e, fuse, ordered, partitioned, stream);
    case GAS_PROG_PAGERANK:
      return launch_generic_gather<progs::PageRank>(e, fuse, ordered, partitioned, stream);
    default: return GAS_OK;  // BFS: gatherMap/gatherReduce are no-ops
  }
}

gas_status_t builtin_apply_only(gas_engine *e, void *stream) {
  const int grid = e->capturing ? 8 * e->num_sms
                                : grid_for(e->n_active, kNT, 8 * e->num_sms);
  switch (e->prog) {
    case GAS_PROG_BFS:
      k_bfs_apply<<<grid, kNT, 0, S(stream)>>>(e->act, e->cnt,
                                                (int32_t *)e->vd, e->ret, e->level,
                                                e->level_from_counters ? 1 : 0);
      break;
    case GAS_PROG_SSSP:
      gasdev::k_apply_only<progs::Sssp><<<grid, kNT, 0, S(stream)>>>(
          e->act, e->cnt, (int32_t *)e->vd,
          e->have_gres ? (const int32_t *)e->gres : nullptr, e->ret);
      break;
    case GAS_PROG_CC:
      gasdev::k_apply_only<progs::Cc><<<grid, kNT, 0, S(stream)>>>(
          e->act, e->cnt, (int32_t *)e->vd,
          e->have_gres ? (const int32_t *)e->gres : nullptr, e->ret);
      break;
    case GAS_PROG_PAGERANK:
      gasdev::k_apply_only<progs::PageRank><<<grid, kNT, 0, S(stream)>>>(
          e->act, e->cnt, (progs::PrVertex *)e->vd,
          e->have_gres ? (const float *)e->gres : nullptr, e->ret);
      break;
    default:
      return gas::fail(GAS_ERR_UNSUPPORTED, "apply: not a built-in program");
  }
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

// commit pending slots, expand, compact; end: the loop control of a
// device-side run.
gas_status_t scatter_common(gas_engine *e, void *stream, const LoopEnd &end) {
  const uint8_t *slot = e->slots_pending ? (const uint8_t *)e->slot : nullptr;
  e->slots_pending = false;
  ExpandCtl *ctl = static_cast<ExpandCtl *>(e->xctl);
  int2 *chunks = static_cast<int2 *>(e->xchunks);
  const int2 *list = static_cast<const int2 *>(e->xlist);
  // the active and chunk counts are only known on the device: fixed grids
  k_expand_mark<<<grid_for(e->nV, kNT, 8 * e->num_sms), kNT, 0, S(stream)>>>(
      e->act, e->cnt, e->ret, e->csr_off, e->csr_dst, e->changed, e->bits, slot,
      (uint8_t *)e->vd, (int)e->vbytes, chunks, list, e->nE, ctl);
  k_expand<<<grid_for(std::max<int64_t>(e->nV, e->nE / 2), kNT, 8 * e->num_sms), kNT, 0,
             S(stream)>>>(e->act, e->cnt, e->ret, e->csr_off, e->csr_dst, e->csc_off, e->csc_src,
                          e->nV, e->nE, e->changed, chunks, ctl,
                          list, e->xlist_n, e->bits);
  CUDA_TRY(cudaGetLastError());
  const int nW = (e->nV + 31) / 32, nb = e->n_cblocks;
  int2 *part = static_cast<int2 *>(e->cpart), *wpart = part + nb;
  const int tile = e->prog == GAS_PROG_USER ? 0 : kBuiltinTile;  // users partition themselves
  k_compact_count<<<nb, kNT, 0, S(stream)>>>(e->bits, e->changed, e->csc_off, nW, e->nE, part,
                                             wpart, ctl, e->cnt);
  if (nb > kCSumBlocks) k_compact_spine<<<1, kNT, 0, S(stream)>>>(part, nb);
  k_compact_write<<<nb, kNT, 0, S(stream)>>>(e->bits, e->csc_off, nW, part, wpart,
                                             nb > kCSumBlocks ? 1 : 0, e->act, e->scan,
                                             e->tpart, tile, e->cnt, end);
  CUDA_TRY(cudaGetLastError());
  e->tpart_valid = tile > 0;
  e->counts_dirty = true;
  e->have_gres = false;
  e->active_full = false;
  return GAS_OK;
}

gas_status_t flush_pending_gather(gas_engine *e, void *stream) {
  if (!e->pending_gather) return GAS_OK;
  e->pending_gather = false;
  if (e->prog == GAS_PROG_USER)
    return gas::fail(GAS_ERR_STATE, "user engine: gather must be launched by the header");
  GAS_TRY(builtin_gather(e, /*fuse=*/false, false, e->tpart_valid, stream));
  e->have_gres = true;
  return GAS_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

const char *gas_status_string(gas_status_t s) {
  switch (s) {
    case GAS_OK: return "ok";
    case GAS_ERR_INVALID: return "invalid argument";
    case GAS_ERR_NOMEM: return "out of memory";
    case GAS_ERR_CUDA: return "CUDA error";
    case GAS_ERR_ITER_CAP: return "iteration cap reached";
    case GAS_ERR_IO: return "I/O error";
    case GAS_ERR_STATE: return "call out of order";
    case GAS_ERR_UNSUPPORTED: return "unsupported";
    case GAS_ERR_DEVICE: return "device-side error";
    case GAS_ERR_TOO_LARGE: return "too large";
  }
  return "unknown status";
}

const char *gas_last_error(void) { return gas::g_err_ptr(); }

const char *gas_version(void) { return "libgas 0.1 (sm_103a)"; }

gas_status_t gas_engine_create(gas_program_t program, gas_engine **out) {
  if (!out) return gas::fail(GAS_ERR_INVALID, "null out");
  if (program < GAS_PROG_BFS || program > GAS_PROG_PAGERANK)
    return gas::fail(GAS_ERR_INVALID, "unknown program %d", (int)program);
  gas_engine *e = new (std::nothrow) gas_engine;
  if (!e) return gas::fail(GAS_ERR_NOMEM, "engine");
  e->prog = program;
  e->vbytes = program_vbytes(program);
  e->gbytes = 4;
  e->ebytes = 4;
  if (const char *pd = getenv("GAS_PULL_DIV")) {
    const int v = atoi(pd);
    if (v > 0) e->pull_div = v;
  }
  *out = e;  // CUDA is first touched by set_graph
  return GAS_OK;
}

gas_status_t gas_engine_create_user(size_t vertex_bytes, size_t gather_bytes,
                                    size_t edge_bytes, gas_engine **out) {
  if (!out || vertex_bytes == 0 || gather_bytes == 0)
    return gas::fail(GAS_ERR_INVALID, "create_user: bad sizes");
  gas_status_t s = gas_engine_create(GAS_PROG_BFS, out);
  if (s != GAS_OK) return s;
  (*out)->prog = GAS_PROG_USER;
  (*out)->vbytes = vertex_bytes;
  (*out)->gbytes = gather_bytes;
  (*out)->ebytes = edge_bytes;
  return GAS_OK;
}

void gas_engine_destroy(gas_engine *e) {
  if (!e) return;
  free_graph(e);
  for (int i = 0; i < 2; ++i)
    if (e->prof_ev[i]) cudaEventDestroy(e->prof_ev[i]);
  if (e->h_cnt) cudaFreeHost(e->h_cnt);
  delete e;
}

gas_status_t gas_engine_set_graph(gas_engine *e, int32_t nV, void *vertex_data,
                                  int64_t nE, const void *edge_data,
                                  const int32_t *srcs, const int32_t *dsts,
                                  void *stream) {
  if (!e || nV < 0 || nE < 0 || (nE > 0 && (!srcs || !dsts)) ||
      (nV > 0 && !vertex_data))
    return gas::fail(GAS_ERR_INVALID, "set_graph: bad arguments");
  if (nE > INT32_MAX || (int64_t)nV + nE + 1 > INT32_MAX)
    return gas::fail(GAS_ERR_TOO_LARGE, "set_graph: V + E must stay below 2^31");
  if (e->prog == GAS_PROG_SSSP && nE > 0 && !edge_data)
    return gas::fail(GAS_ERR_INVALID, "SSSP needs edge weights");
  if (e->prog == GAS_PROG_SSSP) {
    // The SSSP Program's margin (sssp.cu:32-33): gatherZero = INT_MAX - 100000,
    // so dist + w stays below INT_MAX only for weights up to 100000.
    const int32_t *w = static_cast<const int32_t *>(edge_data);
    int bad = 0;  // branch-free over the host's threads (31 M weights: 12 -> 1 ms)
#pragma omp parallel for reduction(| : bad) if (nE > (1 << 18))
    for (int64_t i = 0; i < nE; ++i) bad |= (uint32_t)w[i] > 100000u;
    if (bad) {
      int64_t i = 0;
      while ((uint32_t)w[i] <= 100000u) ++i;
      return gas::fail(GAS_ERR_INVALID,
                       "set_graph: SSSP weight %d of edge %lld outside [0, 100000]", w[i],
                       (long long)i);
    }
  }
  free_graph(e);
  if (!e->h_cnt) {
    int dev = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce == cudaSuccess)
      ce = cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (ce == cudaSuccess)
      ce = cudaMallocHost((void **)&e->h_cnt, sizeof(gas_counters));
    if (ce != cudaSuccess) {
      e->h_cnt = nullptr;
      return gas::fail(GAS_ERR_CUDA, "set_graph: %s", cudaGetErrorString(ce));
    }
  }
  e->nV = nV;
  e->nE = (int32_t)nE;
  e->host_vd = vertex_data;

  // CSC / CSR (stable by edge-list order), edge data permuted into both
  // orders (gpugas.h:1358-1378): on the device for large graphs, by a
  // counting sort on the host otherwise (GAS_GRAPH_BUILD=host|device forces
  // one).
  const size_t eb = e->ebytes;
  const bool have_ed = edge_data && eb > 0;
  const bool want_perms = have_ed && e->prog == GAS_PROG_USER;
  const bool dev_build = gas::device_build_for(nE);
  std::vector<int32_t> csc_off, csc_src, csc_perm, csr_off, csr_dst, csr_perm;
  std::vector<uint8_t> ed_csc, ed_csr;
  if (!dev_build) {
    try {
      csc_off.resize((size_t)nV + 1);
      csc_src.resize(nE); csc_perm.resize(nE);
      csr_off.resize((size_t)nV + 1); csr_dst.resize(nE); csr_perm.resize(nE);
    } catch (...) {
      return gas::fail(GAS_ERR_NOMEM, "set_graph: host arrays");
    }
    GAS_TRY(gas::build_csr_host(nV, nE, dsts, srcs, csc_off.data(),
                                csc_src.data(), csc_perm.data()));
    GAS_TRY(gas::build_csr_host(nV, nE, srcs, dsts, csr_off.data(),
                                csr_dst.data(), csr_perm.data()));
    if (have_ed) {
      try {
        ed_csc.resize((size_t)nE * eb);
        ed_csr.resize((size_t)nE * eb);
      } catch (...) {
        return gas::fail(GAS_ERR_NOMEM, "set_graph: edge data");
      }
      const uint8_t *src = (const uint8_t *)edge_data;
      for (int64_t i = 0; i < nE; ++i) {
        memcpy(&ed_csc[i * eb], src + (size_t)csc_perm[i] * eb, eb);
        memcpy(&ed_csr[i * eb], src + (size_t)csr_perm[i] * eb, eb);
      }
    }
  }

  const size_t V = (size_t)nV, E = (size_t)nE, nW = (V + 31) / 32;
  ArenaPlan plan(e);
  plan.add(&e->csc_off, V + 1);
  plan.add(&e->csr_off, V + 1);
  e->edges_on_host = e->edge_place == GAS_EDGES_HOST;
  if (e->edges_on_host) {
    GAS_TRY(halloc(&e->csc_src, E));
    GAS_TRY(halloc(&e->csr_dst, E));
    if (have_ed) {
      GAS_TRY(halloc((uint8_t **)&e->csc_ed, E * eb));
      GAS_TRY(halloc((uint8_t **)&e->csr_ed, E * eb));
    }
  } else {
    plan.add(&e->csc_src, E);
    plan.add(&e->csr_dst, E);
    if (have_ed) {
      plan.add((uint8_t **)&e->csc_ed, E * eb);
      plan.add((uint8_t **)&e->csr_ed, E * eb);
    }
  }
  plan.add((uint8_t **)&e->vd, V * e->vbytes);
  plan.add(&e->act, V);
  plan.add(&e->scan, V + 1);
  plan.add(&e->ret, V);
  plan.add((uint8_t **)&e->slot, V * e->vbytes);
  plan.add((uint8_t **)&e->gres, V * std::max<size_t>(e->gbytes, 4));
  plan.add(&e->bits, nW);
  plan.add(&e->changed, nW);
  // smallest tile is kNT * 2 items (gather values larger than 16 bytes)
  const int64_t min_tile = kNT * 2;
  e->tile_cap = (int32_t)(((int64_t)V + (int64_t)E + min_tile - 1) / min_tile + 1);
  const size_t tv = std::max<size_t>(e->gbytes, 8);
  plan.add((uint8_t **)&e->tile_first, (size_t)e->tile_cap * tv);
  plan.add((uint8_t **)&e->tile_carry, (size_t)e->tile_cap * tv);
  plan.add(&e->tile_a0, (size_t)e->tile_cap);
  plan.add(&e->tpart, (size_t)e->tile_cap + 2);
  // a row of d > kXLight out-edges lists ceil(d / kXChunk) <= d / kXLight chunks
  plan.add((int2 **)&e->xchunks, E / kXLight + 1);
  plan.add((ExpandCtl **)&e->xctl, 1);
  e->xlist = nullptr;  // in-edges in host memory are not looked through
  if (!e->edges_on_host && !e->graph_only) {
    plan.add((int2 **)&e->xlist, E / kXLight + 1);
    plan.add(&e->xlist_n, 1);
  }
  e->n_cblocks = (int32_t)std::max<size_t>(1, (nW + kCBlockWords - 1) / kCBlockWords);
  // block totals, then the blocks' per-warp totals
  plan.add((int2 **)&e->cpart, (size_t)e->n_cblocks * (1 + kCWarps));
  plan.add(&e->cnt, 1);
  // rows of the CSC with in-edges, for the dense slab passes
  plan.add(&e->ne_vid, V);
  plan.add(&e->ne_end, V);
  e->slab_cap = (int32_t)((E + gasdev::kSlabChunk - 1) / gasdev::kSlabChunk + 1);
  plan.add(&e->slab_dpart, (size_t)e->slab_cap);
  // the push may cut its queue's edges into chunks as small as 64 edges
  plan.add(&e->slab_qpart, (size_t)((E >> gasdev::kSlabChunkMinLog2) + 2));
  plan.add(&e->slab_a0, (size_t)e->slab_cap);
  plan.add((uint8_t **)&e->slab_first, (size_t)e->slab_cap * 8);
  plan.add((uint8_t **)&e->slab_carry, (size_t)e->slab_cap * 8);
  plan.add(&e->slab_fix, (size_t)e->slab_cap);
  plan.add(&e->slab_fix_n, 1);
  plan.add(&e->trace, GAS_TRACE_CAP);
  plan.add(&e->hist, 8);
  plan.add(&e->ne_scratch, (size_t)gas::ne_blocks(nV) + 1);
  if (!e->graph_only && !e->edges_on_host) {
    const gas::SmallBytes sb = gas::bfs_small_bytes(nV, nE), sm = gas::min_small_bytes(nV, nE);
    if (e->prog == GAS_PROG_BFS && sb.all() <= gas::kSmallWithGraph) {
      plan.add((uint8_t **)&e->sb_bits, sb.values);
      plan.add((uint8_t **)&e->sb_ctl, sb.ctl);
      plan.add((uint8_t **)&e->sb_queue, sb.queues);
    }
    if ((e->prog == GAS_PROG_SSSP || e->prog == GAS_PROG_CC) &&
        sm.all() <= gas::kSmallWithGraph) {
      plan.add((uint8_t **)&e->sm_vals, sm.values);
      plan.add((uint8_t **)&e->sm_ctl, sm.ctl);
      plan.add((uint8_t **)&e->sm_queue, sm.queues);
    }
  }
  GAS_TRY(plan.alloc());

  if (dev_build)
    GAS_TRY(gas::build_graph_device(e, srcs, dsts, have_ed ? edge_data : nullptr,
                                    want_perms ? &csc_perm : nullptr,
                                    want_perms ? &csr_perm : nullptr, stream));
  if (want_perms) {
    // a user program may scatter into its edge data: keep what maps the
    // two device copies onto each other and back to the caller's order
    try {
      std::vector<int32_t> inv((size_t)nE);
      for (int64_t i = 0; i < nE; ++i) inv[csc_perm[i]] = (int32_t)i;
      e->h_csr_to_csc.resize((size_t)nE);
      for (int64_t j = 0; j < nE; ++j) e->h_csr_to_csc[j] = inv[csr_perm[j]];
      e->h_csr_perm = csr_perm;
    } catch (...) {
      return gas::fail(GAS_ERR_NOMEM, "set_graph: edge maps");
    }
    e->host_ed = const_cast<void *>(edge_data);
  }

  cudaStream_t st = S(stream);
  if (!dev_build) {
    CUDA_TRY(cudaMemcpyAsync(e->csc_off, csc_off.data(), (V + 1) * 4,
                             cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemcpyAsync(e->csr_off, csr_off.data(), (V + 1) * 4, cudaMemcpyHostToDevice,
                             st));
  }
  if (E && !dev_build) {
    CUDA_TRY(cudaMemcpyAsync(e->csc_src, csc_src.data(), E * 4, cudaMemcpyDefault, st));
    CUDA_TRY(cudaMemcpyAsync(e->csr_dst, csr_dst.data(), E * 4, cudaMemcpyDefault, st));
    if (have_ed) {
      CUDA_TRY(cudaMemcpyAsync(e->csc_ed, ed_csc.data(), E * eb, cudaMemcpyDefault, st));
      CUDA_TRY(cudaMemcpyAsync(e->csr_ed, ed_csr.data(), E * eb, cudaMemcpyDefault, st));
    }
  }
  if (V)
    CUDA_TRY(cudaMemcpyAsync(e->vd, vertex_data, V * e->vbytes, cudaMemcpyHostToDevice, st));
  CUDA_TRY(cudaMemsetAsync(e->bits, 0, nW * 4, st));
  CUDA_TRY(cudaMemsetAsync(e->changed, 0, nW * 4, st));
  if (e->xlist) {
    CUDA_TRY(cudaMemsetAsync(e->xlist_n, 0, sizeof(int32_t), st));
    k_expand_list<<<grid_for(nV, kNT, 8 * e->num_sms), kNT, 0, st>>>(
        e->csc_off, nV, static_cast<int2 *>(e->xlist), e->xlist_n);
  }
  CUDA_TRY(cudaMemsetAsync(e->xctl, 0, sizeof(ExpandCtl), st));
  CUDA_TRY(cudaMemsetAsync(e->slab_fix_n, 0, sizeof(int32_t), st));
  CUDA_TRY(cudaMemsetAsync(e->hist, 0, 8 * sizeof(int32_t), st));
  CUDA_TRY(cudaMemsetAsync(e->trace, 0, GAS_TRACE_CAP * sizeof(gas_trace_record), st));
  CUDA_TRY(cudaMemsetAsync(e->cnt, 0, sizeof(gas_counters), st));
  CUDA_TRY(cudaMemsetAsync(e->ret, 0, V ? V : 1, st));
  int32_t *ne_n = e->ne_scratch + gas::ne_blocks(nV);
  GAS_TRY(gas::build_ne_rows(e, e->ne_scratch, ne_n, st));
  int32_t *h_ne = reinterpret_cast<int32_t *>(e->h_cnt);  // pinned, free until the next run
  CUDA_TRY(cudaMemcpyAsync(h_ne, ne_n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  // the host vectors are released at return: wait for the copies
  CUDA_TRY(cudaStreamSynchronize(st));
  e->n_ne = *h_ne;
  gas::reserve_fast_buffers(e, stream);
  e->n_active = 0;
  e->n_edges = 0;
  e->counts_dirty = false;
  e->tpart_valid = false;
  e->pending_gather = e->have_gres = e->slots_pending = false;
  e->level = 0;
  e->has_graph = true;
  return GAS_OK;
}

gas_status_t gas_engine_set_active(gas_engine *e, int32_t start, int32_t end,
                                   void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "set_active before set_graph");
  if (start < 0 || end < start || end > e->nV)
    return gas::fail(GAS_ERR_INVALID, "set_active: [%d,%d) outside [0,%d)", start, end, e->nV);
  GAS_TRY(flush_pending_gather(e, stream));
  if (e->slots_pending) {
    // an applied but not yet scattered iteration: make its vertex data visible
    k_commit<<<grid_for(e->n_active, kNT, 8 * e->num_sms), kNT, 0, S(stream)>>>(
        e->act, e->cnt, (const uint8_t *)e->slot, (uint8_t *)e->vd, (int)e->vbytes);
    CUDA_TRY(cudaGetLastError());
    e->slots_pending = false;
  }
  const int n = end - start;
  k_set_range<<<grid_for((int64_t)n + 1, kNT, 8 * e->num_sms), kNT, 0, S(stream)>>>(
      start, n, e->csc_off, e->act, e->scan, e->cnt, &static_cast<ExpandCtl *>(e->xctl)->wait);
  CUDA_TRY(cudaGetLastError());
  e->tpart_valid = false;
  e->n_active = n;
  e->n_edges = n ? e->nE : 0;  // at most: it sizes the first gather's grid
  e->counts_dirty = false;
  e->active_full = start == 0 && end == e->nV;
  return GAS_OK;
}

gas_status_t gas_engine_count_active(gas_engine *e, int32_t *n_active) {
  if (!e || !n_active) return gas::fail(GAS_ERR_INVALID, "null argument");
  if (e->counts_dirty) GAS_TRY(sync_counts(e, nullptr));
  *n_active = e->n_active;
  return GAS_OK;
}

gas_status_t gas_engine_gather(gas_engine *e, int32_t have_gather, void *stream) {
  (void)stream;
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "gather before set_graph");
  if (e->prog == GAS_PROG_USER)
    return gas::fail(GAS_ERR_UNSUPPORTED, "user programs gather through gpugas.h");
  if (e->counts_dirty) GAS_TRY(sync_counts(e, stream));
  e->pending_gather = have_gather != 0 && e->prog != GAS_PROG_BFS;
  e->have_gres = false;
  return GAS_OK;
}

gas_status_t gas_engine_apply(gas_engine *e, void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "apply before set_graph");
  if (e->prog == GAS_PROG_USER)
    return gas::fail(GAS_ERR_UNSUPPORTED, "user programs apply through gpugas.h");
  if (e->counts_dirty) GAS_TRY(sync_counts(e, stream));
  if (e->n_active == 0) return GAS_OK;
  if (e->pending_gather) {
    e->pending_gather = false;
    GAS_TRY(builtin_gather(e, /*fuse=*/true, false, e->tpart_valid, stream));
    e->slots_pending = true;
    return GAS_OK;
  }
  return builtin_apply_only(e, stream);
}

gas_status_t gas_engine_scatter_activate(gas_engine *e, int32_t have_scatter,
                                         void *stream) {
  (void)have_scatter;
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "scatter before set_graph");
  if (e->counts_dirty) GAS_TRY(sync_counts(e, stream));
  GAS_TRY(flush_pending_gather(e, stream));
  return scatter_common(e, stream, LoopEnd{});
}

gas_status_t gas_engine_next_iter(gas_engine *e, int32_t *n_active, void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "next_iter before set_graph");
  if (e->counts_dirty) GAS_TRY(sync_counts(e, stream));
  if (n_active) *n_active = e->n_active;
  return GAS_OK;
}

gas_status_t gas_engine_get_results(gas_engine *e, void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "get_results before set_graph");
  GAS_TRY(flush_pending_gather(e, stream));
  if (e->slots_pending) {
    k_commit<<<grid_for(e->n_active, kNT, 8 * e->num_sms), kNT, 0, S(stream)>>>(
        e->act, e->cnt, (const uint8_t *)e->slot, (uint8_t *)e->vd, (int)e->vbytes);
    CUDA_TRY(cudaGetLastError());
    e->slots_pending = false;
  }
  if (e->nV && e->host_vd)
    CUDA_TRY(cudaMemcpyAsync(e->host_vd, e->vd, (size_t)e->nV * e->vbytes,
                             cudaMemcpyDeviceToHost, S(stream)));
  CUDA_TRY(cudaStreamSynchronize(S(stream)));
  if (e->edges_dirty && e->host_ed && e->nE) {
    // edge data a user scatter changed, back into the caller's order
    const size_t eb = e->ebytes;
    std::vector<uint8_t> tmp;
    try {
      tmp.resize((size_t)e->nE * eb);
    } catch (...) {
      return gas::fail(GAS_ERR_NOMEM, "get_results: edge data");
    }
    CUDA_TRY(cudaMemcpyAsync(tmp.data(), e->csr_ed, tmp.size(), cudaMemcpyDefault,
                             S(stream)));
    CUDA_TRY(cudaStreamSynchronize(S(stream)));
    uint8_t *dst = static_cast<uint8_t *>(e->host_ed);
    for (int32_t j = 0; j < e->nE; ++j)
      memcpy(dst + (size_t)e->h_csr_perm[j] * eb, &tmp[(size_t)j * eb], eb);
    e->edges_dirty = false;
  }
  return GAS_OK;
}

gas_status_t gas_engine_set_edge_placement(gas_engine *e, gas_edge_placement_t where) {
  if (!e) return gas::fail(GAS_ERR_INVALID, "null engine");
  if (where != GAS_EDGES_DEVICE && where != GAS_EDGES_HOST)
    return gas::fail(GAS_ERR_INVALID, "unknown edge placement %d", (int)where);
  e->edge_place = where;
  return GAS_OK;
}

gas_status_t gas_engine_download_graph(gas_engine *e, int32_t *csc_off, int32_t *csc_src,
                                       int32_t *csr_off, int32_t *csr_dst, void *csc_ed,
                                       void *csr_ed, void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  const size_t V1 = (size_t)e->nV + 1, E = (size_t)e->nE, eb = e->ebytes;
  cudaStream_t st = S(stream);
  const struct {
    void *dst;
    const void *src;
    size_t bytes;
  } cp[] = {{csc_off, e->csc_off, V1 * 4}, {csc_src, e->csc_src, E * 4},
            {csr_off, e->csr_off, V1 * 4}, {csr_dst, e->csr_dst, E * 4},
            {csc_ed, e->csc_ed, E * eb}, {csr_ed, e->csr_ed, E * eb}};
  for (const auto &c : cp)
    if (c.dst && c.src && c.bytes)
      CUDA_TRY(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDefault, st));
  CUDA_TRY(cudaStreamSynchronize(st));
  return GAS_OK;
}

gas_status_t gas_engine_prepare_scatter(gas_engine *e, const int32_t **csr_to_csc,
                                        void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "scatter before set_graph");
  if (e->prog != GAS_PROG_USER)
    return gas::fail(GAS_ERR_UNSUPPORTED, "prepare_scatter is for user programs");
  if (e->counts_dirty) GAS_TRY(sync_counts(e, stream));
  if (e->slots_pending) {
    k_commit<<<grid_for(e->n_active, kNT, 8 * e->num_sms), kNT, 0, S(stream)>>>(
        e->act, e->cnt, (const uint8_t *)e->slot, (uint8_t *)e->vd, (int)e->vbytes);
    CUDA_TRY(cudaGetLastError());
    e->slots_pending = false;
  }
  const bool have = e->csr_ed && e->nE > 0 && !e->h_csr_to_csc.empty();
  if (have && !e->csr_to_csc) {
    GAS_TRY(dalloc(&e->csr_to_csc, (size_t)e->nE));
    CUDA_TRY(cudaMemcpyAsync(e->csr_to_csc, e->h_csr_to_csc.data(), (size_t)e->nE * 4,
                             cudaMemcpyHostToDevice, S(stream)));
  }
  if (csr_to_csc) *csr_to_csc = have ? e->csr_to_csc : nullptr;
  e->edges_dirty = e->edges_dirty || have;
  return GAS_OK;
}

gas_status_t gas_engine_set_iteration(gas_engine *e, int32_t level) {
  if (!e) return gas::fail(GAS_ERR_INVALID, "null engine");
  e->level = level;
  return GAS_OK;
}

gas_status_t gas_engine_run(gas_engine *e, int32_t *iterations, void *stream) {
  if (!e || !e->has_graph) return gas::fail(GAS_ERR_STATE, "run before set_graph");
  if (e->prog == GAS_PROG_USER)
    return gas::fail(GAS_ERR_UNSUPPORTED, "user programs run through gpugas.h");
  int32_t it = 0, n = 0;
  GAS_TRY(gas_engine_count_active(e, &n));
  while (n) {
    GAS_TRY(gas_engine_gather(e, 1, stream));
    GAS_TRY(gas_engine_apply(e, stream));
    GAS_TRY(gas_engine_scatter_activate(e, 1, stream));
    GAS_TRY(gas_engine_next_iter(e, &n, stream));
    ++it;
    if (e->prog == GAS_PROG_BFS) e->level = it;
  }
  if (iterations) *iterations = it;
  return GAS_OK;
}

gas_status_t gas_engine_vertex_data_device(gas_engine *e, void **ptr) {
  if (!e || !ptr || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  *ptr = e->vd;
  return GAS_OK;
}

gas_status_t gas_engine_upload_vertex_data(gas_engine *e, const void *host,
                                           void *stream) {
  if (!e || !host || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  CUDA_TRY(cudaMemcpyAsync(e->vd, host, (size_t)e->nV * e->vbytes,
                           cudaMemcpyDefault, S(stream)));
  return GAS_OK;
}

gas_status_t gas_engine_download_vertex_data(gas_engine *e, void *host,
                                             void *stream) {
  if (!e || !host || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  CUDA_TRY(cudaMemcpyAsync(host, e->vd, (size_t)e->nV * e->vbytes,
                           cudaMemcpyDefault, S(stream)));
  CUDA_TRY(cudaStreamSynchronize(S(stream)));
  return GAS_OK;
}

gas_status_t gas_engine_download_vertex_data_async(gas_engine *e, void *dst,
                                                   void *stream) {
  if (!e || !dst || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  CUDA_TRY(cudaMemcpyAsync(dst, e->vd, (size_t)e->nV * e->vbytes, cudaMemcpyDefault,
                           S(stream)));
  return GAS_OK;
}

gas_status_t gas_engine_view_get(gas_engine *e, gas_engine_view *v) {
  if (!e || !v || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  v->nV = e->nV;
  v->nE = e->nE;
  v->csc_off = e->csc_off;
  v->csc_src = e->csc_src;
  v->csc_ed = e->csc_ed;
  v->csr_off = e->csr_off;
  v->csr_dst = e->csr_dst;
  v->csr_ed = e->csr_ed;
  v->vertex_data = e->vd;
  v->active = e->act;
  v->active_scan = e->scan;
  v->apply_ret = e->ret;
  v->slot = e->slot;
  v->gather_tmp = e->gres;
  v->tile_first = e->tile_first;
  v->tile_carry = e->tile_carry;
  v->tile_a0 = e->tile_a0;
  v->tile_part = e->tpart;
  v->tile_cap = e->tile_cap;
  v->num_sms = e->num_sms;
  v->counters = e->cnt;
  return GAS_OK;
}

gas_status_t gas_engine_note_applied(gas_engine *e, int32_t wrote_slots) {
  if (!e) return gas::fail(GAS_ERR_INVALID, "null engine");
  e->slots_pending = wrote_slots != 0;
  return GAS_OK;
}

gas_status_t gas_engine_set_profiling(gas_engine *e, int32_t on) {
  if (!e) return gas::fail(GAS_ERR_INVALID, "null engine");
  if (on) {
    for (int i = 0; i < 2; ++i)
      if (!e->prof_ev[i]) CUDA_TRY(cudaEventCreate(&e->prof_ev[i]));
  }
  e->profiling = on != 0;
  return GAS_OK;
}

gas_status_t gas_engine_get_profile(gas_engine *e, gas_kernel_profile *out,
                                    int32_t reset) {
  if (!e || !out) return gas::fail(GAS_ERR_INVALID, "null argument");
  *out = e->prof;
  if (reset) e->prof = gas_kernel_profile{};
  return GAS_OK;
}

gas_status_t gas_engine_read_counters(gas_engine *e, gas_counters *out,
                                      void *stream) {
  if (!e || !out || !e->has_graph) return gas::fail(GAS_ERR_STATE, "no graph");
  GAS_TRY(sync_counts(e, stream));
  *out = *e->h_cnt;
  return GAS_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Schedules, precision PageRank (gas_engine_run_schedule and friends) live in
// gas_runs.cu; they reach the engine through these accessors.
// ---------------------------------------------------------------------------
namespace gas {

void prof_begin(gas_engine *e, cudaStream_t s, int kind, int64_t bytes) {
  if (!e->profiling || e->in_graph || !e->prof_ev[0]) return;
  cudaEventRecord(e->prof_ev[0], s);
  e->prof_kind = kind;
  e->prof_bytes_pending = bytes;
}

void prof_end(gas_engine *e, cudaStream_t s) {
  if (e->prof_kind < 0) return;
  cudaEventRecord(e->prof_ev[1], s);
}

void prof_collect(gas_engine *e) {
  if (e->prof_kind < 0) return;
  float ms = 0.f;
  if (cudaEventSynchronize(e->prof_ev[1]) == cudaSuccess &&
      cudaEventElapsedTime(&ms, e->prof_ev[0], e->prof_ev[1]) == cudaSuccess) {
    gas_kernel_profile &p = e->prof;
    if (e->prof_kind == kProfPush) {
      p.push_ms += ms; p.push_bytes += e->prof_bytes_pending; ++p.push_launches;
    } else if (e->prof_kind == kProfPull) {
      p.pull_ms += ms; p.pull_bytes += e->prof_bytes_pending; ++p.pull_launches;
    } else {
      p.pagerank_ms += ms; p.pagerank_bytes += e->prof_bytes_pending; ++p.pagerank_launches;
    }
  }
  e->prof_kind = -1;
}

gas_status_t engine_scatter_loop(gas_engine *e, cudaGraphConditionalHandle h, void *stream) {
  return scatter_common(e, stream, LoopEnd{1, e->in_graph ? 1 : 0, h});
}
gas_status_t engine_sync_counts(gas_engine *e, void *stream) {
  return sync_counts(e, stream);
}
int engine_grid(int64_t work_items, int per_block, int cap) {
  return grid_for(work_items, per_block, cap);
}
int engine_partition_grid(gas_engine *e, int64_t items, int tile) {
  const int cap = 2 * e->num_sms;
  if (e->capturing || items < 0) return cap;
  return grid_for((items + tile - 1) / tile + 1, 256, cap);
}

gas_status_t engine_gather_apply(gas_engine *e, void *stream) {
  // captured once and replayed on any active set: partitions itself
  GAS_TRY(builtin_gather(e, true, false, false, stream));
  e->slots_pending = true;
  return GAS_OK;
}
gas_status_t engine_apply_only(gas_engine *e, void *stream) {
  return builtin_apply_only(e, stream);
}
gas_status_t engine_commit(gas_engine *e, void *stream) {
  const int g = e->capturing ? 8 * e->num_sms
                             : grid_for(e->n_active, kNT, 8 * e->num_sms);
  k_commit<<<g, kNT, 0, S(stream)>>>(e->act, e->cnt, (const uint8_t *)e->slot,
                                     (uint8_t *)e->vd, (int)e->vbytes);
  CUDA_TRY(cudaGetLastError());
  e->slots_pending = false;
  return GAS_OK;
}

gas_status_t engine_generic_iteration(gas_engine *e, bool ordered,
                                      cudaGraphConditionalHandle h, void *stream) {
  if (e->prog == GAS_PROG_BFS) {
    GAS_TRY(builtin_apply_only(e, stream));
  } else {
    GAS_TRY(builtin_gather(e, true, ordered, /*partitioned=*/true, stream));
    e->slots_pending = true;
  }
  return engine_scatter_loop(e, h, stream);
}

gas_status_t engine_partition(gas_engine *e, void *stream) {
  const SegSource src = gasdev::frontier_source(
      e->act, e->scan, e->csc_off, &e->cnt->n_active, &e->cnt->n_edges, e->tpart);
  gasdev::k_partition<kBuiltinTile, false>
      <<<engine_partition_grid(e, (int64_t)e->n_active + e->n_edges, kBuiltinTile), 256, 0,
         S(stream)>>>(src, e->tpart);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

int engine_scatter_kernels(const gas_engine *e) { return e->n_cblocks > kCSumBlocks ? 5 : 4; }
}  // namespace gas
