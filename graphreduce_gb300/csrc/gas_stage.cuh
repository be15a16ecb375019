// gas_stage.cuh -- the frontier queue of the persistent kernels (the small-
// graph BFS, SSSP and CC): CTAs of 1,024 threads collect new members in shared
// memory and append them to a global queue after their edges, one atomic per
// 1,024.  A queue holds light members (few out-edges, none included) as one
// entry each and the others as several entries of at most kEntryEdges edges,
// so that any run of entries is balanced.  Not installed.
#ifndef GAS_STAGE_CUH_
#define GAS_STAGE_CUH_

#include "gas_grid.cuh"

namespace gasstage {

constexpr int kNT = 1024;
constexpr int kWarps = kNT / 32;
constexpr int kLight = 32;        // out-edges of a light member
constexpr int kEntryEdges = 128;
constexpr int kHeavyMost = 8;     // heavy entries a warp takes at once (1: 20 %
                                  // slower on R-MAT 4 M, 32: 8 % on 1 M)
constexpr int kStage = 4096;      // members a CTA collects before it appends directly
// Entries of a queue, and its members' out-edges and number.
struct Count {
  int light, heavy, edges, members;
};

__device__ __forceinline__ int32_t ld_edge(const int32_t *p) {
  int32_t v;
  asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// A queue: light members (at most kLight out-edges, none included), one entry
// each, and the others as heavy entries of kEntryEdges edges.
struct Queue {
  int4 *light, *heavy;  // (vertex, CSR position, edges)
};

// Light entries, heavy entries and out-edges of one member per lane (v < 0:
// none), their inclusive sums over the warp, and the warp's members.
struct Member {
  int v, off, deg, nl, nh;
  int il, ih, ie, n;
};

__device__ __forceinline__ Member member(int v, const int32_t *csr_off) {
  Member m;
  m.v = v;
  m.off = v >= 0 ? __ldg(csr_off + v) : 0;
  m.deg = v >= 0 ? __ldg(csr_off + v + 1) - m.off : 0;
  m.nl = v >= 0 && m.deg <= kLight ? 1 : 0;
  m.nh = m.deg > kLight ? (m.deg + kEntryEdges - 1) / kEntryEdges : 0;
  m.il = __popc(__ballot_sync(0xffffffffu, m.nl) & (0xffffffffu >> (31 - (threadIdx.x & 31))));
  m.ih = gasgrid::warp_incl_sum(m.nh);
  m.ie = gasgrid::warp_incl_sum(m.deg);
  m.n = __popc(__ballot_sync(0xffffffffu, v >= 0));
  return m;
}

// Room for nl light and nh heavy entries of n members with ne edges.
__device__ __forceinline__ int2 reserve(Count *c, int nl, int nh, int ne, int n) {
  int2 at = make_int2(0, 0);
  if (nh) at.y = atomicAdd(&c->heavy, nh);
  if (nl) at.x = atomicAdd(&c->light, nl);
  if (ne) atomicAdd(&c->edges, ne);
  if (n) atomicAdd(&c->members, n);
  return at;
}

// All lanes of the warp call.  A hub's entries are written by the whole warp:
// one lane writing 1,000 of them kept its CTA 40 us.
__device__ __forceinline__ void write_entries(const Queue &q, const Member &m, int al, int ah) {
  constexpr int kFew = 4;
  if (m.nl) q.light[al + m.il - 1] = make_int4(m.v, m.off, m.deg, 0);
  ah += m.ih - m.nh;
  if (m.nh <= kFew)
    for (int e = 0; e < m.nh; ++e)
      q.heavy[ah + e] = make_int4(m.v, m.off + e * kEntryEdges,
                                  min(m.deg - e * kEntryEdges, kEntryEdges), 0);
  for (unsigned big = __ballot_sync(0xffffffffu, m.nh > kFew); big; big &= big - 1) {
    const int l = __ffs(big) - 1;
    const int v = __shfl_sync(0xffffffffu, m.v, l), off = __shfl_sync(0xffffffffu, m.off, l);
    const int deg = __shfl_sync(0xffffffffu, m.deg, l), n = __shfl_sync(0xffffffffu, m.nh, l);
    const int at = __shfl_sync(0xffffffffu, ah, l);
    for (int e = threadIdx.x & 31; e < n; e += 32)
      q.heavy[at + e] =
          make_int4(v, off + e * kEntryEdges, min(deg - e * kEntryEdges, kEntryEdges), 0);
  }
}

// The warp's number when a queue is dealt out: consecutive ones are in
// different CTAs, so that few entries (and the members they find) spread
// over all SMs.
__device__ __forceinline__ int dealt_warp() {
  return (int)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
}

struct Stage {
  int n;  // members offered this iteration (those past kStage went out directly)
  int v[kStage];
  int wl[kWarps], wh[kWarps], we[kWarps], wn[kWarps];
  int2 base;
};

// All lanes of the warp call; v[h] >= 0: a new member.
template <int K>
__device__ __forceinline__ void offer(Stage &st, const int (&v)[K], const int32_t *csr_off,
                                      const Queue &q, Count *c) {
  const int lane = threadIdx.x & 31;
  unsigned m[K];
  int n = 0;
#pragma unroll
  for (int h = 0; h < K; ++h) {
    m[h] = __ballot_sync(0xffffffffu, v[h] >= 0);
    n += __popc(m[h]);
  }
  if (!n) return;
  int at = 0;
  if (lane == 0) at = atomicAdd(&st.n, n);
  at = __shfl_sync(0xffffffffu, at, 0);
  const bool over = at + n > kStage;  // warp-uniform
#pragma unroll
  for (int h = 0; h < K; ++h) {
    const int pos = at + __popc(m[h] & ((1u << lane) - 1u));
    at += __popc(m[h]);
    if (!over) {
      if (v[h] >= 0) st.v[pos] = v[h];
    } else if (m[h]) {  // no room left in the stage: straight to the queue
      if (v[h] >= 0 && pos < kStage) st.v[pos] = -1;
      const Member mb = member(v[h], csr_off);
      int2 to = make_int2(0, 0);
      if (lane == 31) to = reserve(c, mb.il, mb.ih, mb.ie, mb.n);
      write_entries(q, mb, __shfl_sync(0xffffffffu, to.x, 31),
                    __shfl_sync(0xffffffffu, to.y, 31));
    }
  }
}

// The collected members to the queue (every thread of the CTA calls).
__device__ __forceinline__ void flush(Stage &st, const int32_t *csr_off, const Queue &q,
                                      Count *c) {
  __syncthreads();
  const int n = min(st.n, kStage);
  __syncthreads();        // every warp has the count before any goes on
  if (n == 0) return;     // CTA-uniform
  if (threadIdx.x == 0) st.n = 0;  // before the next offers: a barrier follows
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (n <= 32) {  // one warp's worth: the rest of the CTA waits at the caller's barrier
    if (warp == 0) {
      const Member m = member(lane < n ? st.v[lane] : -1, csr_off);
      int2 at = make_int2(0, 0);
      if (lane == 31) at = reserve(c, m.il, m.ih, m.ie, m.n);
      write_entries(q, m, __shfl_sync(0xffffffffu, at.x, 31), __shfl_sync(0xffffffffu, at.y, 31));
    }
    __syncthreads();
    return;
  }
  for (int i0 = 0; i0 < n; i0 += kNT) {  // CTA-uniform
    const Member m = member(i0 + (int)threadIdx.x < n ? st.v[i0 + threadIdx.x] : -1, csr_off);
    if (lane == 31) {
      st.wl[warp] = m.il;
      st.wh[warp] = m.ih;
      st.we[warp] = m.ie;
      st.wn[warp] = m.n;
    }
    __syncthreads();
    if (warp == 0) {
      const int l = st.wl[lane], h = st.wh[lane];
      const int il = gasgrid::warp_incl_sum(l), ih = gasgrid::warp_incl_sum(h);
      const int ie = gasgrid::warp_incl_sum(st.we[lane]);
      const int in = __reduce_add_sync(0xffffffffu, st.wn[lane]);
      st.wl[lane] = il - l;
      st.wh[lane] = ih - h;
      if (lane == 31) st.base = reserve(c, il, ih, ie, in);
    }
    __syncthreads();
    write_entries(q, m, st.base.x + st.wl[warp], st.base.y + st.wh[warp]);
    __syncthreads();
  }
}

// Heavy entries of a queue: at most ceil(deg / kEntryEdges) <= deg / kLight
// per member.
inline size_t heavy_cap(size_t n_edges) { return n_edges / kLight + 1; }

// A warp's entries (start and edges per lane, 0: none) laid end to end, those
// with edges in consecutive lanes: row k's first place and CSR position -
// place, and what val it carries.  Returns the edges.
struct Rows {
  bool ok;
  int excl, shift, val;
};

__device__ __forceinline__ int lay_out(int start, int deg, int val, int (*s_row)[3], Rows &r) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned rb = __ballot_sync(FULL, deg > 0);
  const int incl = gasgrid::warp_incl_sum(deg);
  if (deg > 0) {
    int *s = s_row[__popc(rb & ((1u << lane) - 1u))];
    s[0] = incl - deg;
    s[1] = start - (incl - deg);
    s[2] = val;
  }
  __syncwarp();
  r.ok = lane < __popc(rb);
  r.excl = r.ok ? s_row[lane][0] : 0;
  r.shift = r.ok ? s_row[lane][1] : 0;
  r.val = r.ok ? s_row[lane][2] : 0;
  __syncwarp();
  return __shfl_sync(FULL, incl, 31);
}

// The row of this lane's edge in the round of 32 that begins at place r0: the
// last row starting at or before r0, plus the rows that start inside.
__device__ __forceinline__ int row_of(const Rows &r, int r0) {
  constexpr unsigned FULL = 0xffffffffu;
  const int row0 = __popc(__ballot_sync(FULL, r.ok && r.excl <= r0)) - 1;
  const int d = r.excl - r0;
  const unsigned starts = __reduce_or_sync(FULL, (r.ok && d >= 1 && d < 32) ? (1u << d) : 0u);
  return min(31, row0 + __popc(starts & ((2u << (threadIdx.x & 31)) - 1u)));
}

}  // namespace gasstage

#endif  // GAS_STAGE_CUH_
