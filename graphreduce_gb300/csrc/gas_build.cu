// gas_build.cu -- CSR and CSC construction on the device (the work of
// edgeListToCSR / edgeListToCSC, util.cuh:80-121, done by setGraph at
// gpugas.h:1314-1503, moved off the host).
//
// The edge list goes to the device once.  Each of the two orders is a stable
// LSD radix sort of the edge indices by key (source for CSR, destination for
// CSC), 8 bits per pass over the bits the vertex count needs, followed by
// row offsets read off the sorted keys and gathers of the other endpoint and
// of the edge data; an order the edge list is in already (sorted by source,
// as .gr files and the generators give it) needs no sort, only copies.
// Stability makes the result identical to the host build (edges of one key
// keep their edge-list order).
//
// One pass over n keys: k_rs_hist counts the digits of every 8192-key tile
// (digit-major table [256][tiles]); an exclusive scan of the table gives every
// (digit, tile) its output base; k_rs_scatter ranks the tile's keys stably (a
// warp its own run of keys, by match masks and per-warp digit counts), orders
// them in shared memory and writes them out digit run by digit run, 32 keys
// of a run on average, so the stores are mostly whole lines.  Bound by memory
// (20 bytes per key and pass).  30 M edges, 1 M vertices: three passes of
// 0.36 ms; 4-bit digits, 2048-key tiles and counts per thread took five of
// 0.46 ms, for both orders.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "gas.h"
#include "gas_engine_impl.h"
#include "gas_internal.h"

namespace {

inline cudaStream_t S(void *s) { return (cudaStream_t)s; }

constexpr int kRBits = 8;
constexpr int kRBins = 1 << kRBits;
constexpr int kRThreads = 256;               // scans and the like
constexpr int kSThreads = 512;               // sort kernels
constexpr int kSWarps = kSThreads / 32;
constexpr int kSItems = 16;
constexpr int kRTile = kSThreads * kSItems;  // keys per tile
constexpr int kScanItems = 16;
constexpr int kScanTile = kRThreads * kScanItems;  // entries per scan block

__device__ __forceinline__ int rs_digit(int32_t k, int shift) {
  return (int)(((uint32_t)k >> shift) & (kRBins - 1));
}

// Exclusive CTA scan of one int per thread (kRThreads threads).
__device__ __forceinline__ int cta_scan_excl(int v, int *total) {
  __shared__ int s_w[kRThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += o;
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  int pre = 0, tot = 0;
  for (int w = 0; w < kRThreads / 32; ++w) {
    if (w < warp) pre += s_w[w];
    tot += s_w[w];
  }
  __syncthreads();
  *total = tot;
  return pre + x - v;
}

// What the edge list is like: (index + 1) of the largest edge with an id
// outside [0, nV), and whether it is out of order by a or by b.
struct EdgeFlags {
  int32_t bad, a_unsorted, b_unsorted;
};

__global__ void k_check_edges(const int32_t *a, const int32_t *b, int n, int nV, EdgeFlags *f) {
  bool ua = false, ub = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int32_t x = a[i], y = b[i];
    if (x < 0 || x >= nV || y < 0 || y >= nV) atomicMax(&f->bad, i + 1);
    if (i > 0) {
      ua |= a[i - 1] > x;
      ub |= b[i - 1] > y;
    }
  }
  if (__any_sync(0xffffffffu, ua) && (threadIdx.x & 31) == 0) f->a_unsorted = 1;
  if (__any_sync(0xffffffffu, ub) && (threadIdx.x & 31) == 0) f->b_unsorted = 1;
}

__global__ void __launch_bounds__(kSThreads)
    k_rs_hist(const int32_t *keys, int n, int shift, int ntiles, int32_t *hist) {
  __shared__ int c[kRBins];
  for (int k = threadIdx.x; k < kRBins; k += kSThreads) c[k] = 0;
  __syncthreads();
  const int base = blockIdx.x * kRTile;
#pragma unroll
  for (int j = 0; j < kSItems; ++j) {
    const long long i = (long long)base + j * kSThreads + threadIdx.x;
    if (i < n) atomicAdd(&c[rs_digit(keys[i], shift)], 1);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kRBins; k += kSThreads)
    hist[(size_t)k * ntiles + blockIdx.x] = c[k];
}

struct SortSmem {
  int32_t key[kRTile];
  int32_t val[kRTile];
  int32_t cnt[kSWarps][kRBins];  // per warp: counts, then offsets inside the digit
  int32_t dstart[kRBins];        // first tile position of a digit
  int32_t gbase[kRBins];
  int32_t wsum[kRBins / 32];
};

__global__ void __launch_bounds__(kSThreads)
    k_rs_scatter(const int32_t *kin, const int32_t *vin, int32_t *kout, int32_t *vout, int n,
                 int shift, int ntiles, const int32_t *ghist) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  SortSmem &sm = *reinterpret_cast<SortSmem *>(s_raw);
  constexpr unsigned FULL = 0xffffffffu;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int base = blockIdx.x * kRTile;
  const int nvalid = min(kRTile, n - base);
  // warp w's keys are tile items [w * 512, (w + 1) * 512), item by item over
  // its lanes, so (item, lane) order is tile order and the ranks are stable
  const int first = warp * (32 * kSItems) + lane;
  int32_t k[kSItems], v[kSItems];
#pragma unroll
  for (int j = 0; j < kSItems; ++j) {
    const int i = first + 32 * j;
    k[j] = i < nvalid ? kin[base + i] : -1;
    v[j] = i < nvalid ? (vin ? vin[base + i] : base + i) : 0;
  }
  for (int c = t; c < kSWarps * kRBins; c += kSThreads) (&sm.cnt[0][0])[c] = 0;
  for (int d = t; d < kRBins; d += kSThreads) sm.gbase[d] = ghist[(size_t)d * ntiles + blockIdx.x];
  __syncthreads();
  int rank[kSItems];
#pragma unroll
  for (int j = 0; j < kSItems; ++j) {
    const bool ok = first + 32 * j < nvalid;
    const int d = ok ? rs_digit(k[j], shift) : kRBins;
    const unsigned same = __match_any_sync(FULL, d);
    const int leader = __ffs(same) - 1;
    int at = 0;
    if (ok && lane == leader) {
      at = sm.cnt[warp][d];
      sm.cnt[warp][d] = at + __popc(same);
    }
    rank[j] = __shfl_sync(FULL, at, leader) + __popc(same & ((1u << lane) - 1u));
    __syncwarp();
  }
  __syncthreads();
  // offsets of the warps inside each digit, then of the digits in the tile
  int run = 0, incl = 0;
  if (t < kRBins) {
#pragma unroll
    for (int w = 0; w < kSWarps; ++w) {
      const int c = sm.cnt[w][t];
      sm.cnt[w][t] = run;
      run += c;
    }
    incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) sm.wsum[warp] = incl;
  }
  __syncthreads();
  if (t < kRBins) {
    int pre = incl - run;
    for (int w = 0; w < warp; ++w) pre += sm.wsum[w];
    sm.dstart[t] = pre;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSItems; ++j) {
    if (first + 32 * j < nvalid) {
      const int d = rs_digit(k[j], shift);
      const int p = sm.dstart[d] + sm.cnt[warp][d] + rank[j];
      sm.key[p] = k[j];
      sm.val[p] = v[j];
    }
  }
  __syncthreads();
  // consecutive tile positions of one digit are consecutive output positions
#pragma unroll
  for (int j = 0; j < kSItems; ++j) {
    const int p = j * kSThreads + t;
    if (p < nvalid) {
      const int32_t key = sm.key[p];
      const int d = rs_digit(key, shift);
      const int g = sm.gbase[d] + (p - sm.dstart[d]);
      kout[g] = key;
      vout[g] = sm.val[p];
    }
  }
}

// Generic exclusive scan of n int32 in place: per-block sums, one block over
// the sums, per-block downsweep.
__global__ void __launch_bounds__(kRThreads)
    k_scan_reduce(const int32_t *a, int n, int32_t *part) {
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += base + k < n ? a[base + k] : 0;
  int total;
  cta_scan_excl(s, &total);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kRThreads) k_scan_spine(int32_t *part, int nb) {
  __shared__ int s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < nb; b0 += kRThreads) {
    const int i = b0 + threadIdx.x;
    const int v = i < nb ? part[i] : 0;
    int total;
    const int e = cta_scan_excl(v, &total);
    const int c = s_carry;
    if (i < nb) part[i] = c + e;
    __syncthreads();
    if (threadIdx.x == 0) s_carry = c + total;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kRThreads)
    k_scan_down(int32_t *a, int n, const int32_t *part) {
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < n ? a[base + k] : 0;
    s += v[k];
  }
  int total;
  int pre = cta_scan_excl(s, &total) + part[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) a[base + k] = pre;
    pre += v[k];
  }
}

// Row offsets from sorted keys: off[v] = first position with key >= v.
__global__ void k_offsets_from_sorted(const int32_t *keys, int n, int nV, int32_t *off) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
    const int lo = i == 0 ? 0 : keys[i - 1] + 1;  // first row starting here
    const int hi = i == n ? nV : keys[i];          // last row starting here
    for (int v = lo; v <= hi; ++v) off[v] = i;
  }
}

__global__ void k_gather_i32(const int32_t *src, const int32_t *perm, int n, int32_t *out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = src[perm[i]];
}

// Edge data of w 32-bit words per edge, or of eb bytes when eb % 4 != 0.
__global__ void k_gather_rec(const uint8_t *src, const int32_t *perm, int n, int eb,
                             uint8_t *out) {
  const size_t total = (size_t)n * eb;
  if (eb % 4 == 0) {
    const int w = eb / 4;
    const uint32_t *s = reinterpret_cast<const uint32_t *>(src);
    uint32_t *o = reinterpret_cast<uint32_t *>(out);
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < (size_t)n * w;
         k += (size_t)gridDim.x * blockDim.x)
      o[k] = s[(size_t)perm[k / w] * w + k % w];
  } else {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total;
         k += (size_t)gridDim.x * blockDim.x)
      out[k] = src[(size_t)perm[k / eb] * eb + k % eb];
  }
}

// Rows with in-edges, in vertex order: counts per block of kScanTile rows,
// then (after a scan) the rows' vertices and in-edge ends.
__device__ __forceinline__ int ne_flags(const int32_t *off, int nV, int v0, unsigned &m) {
  m = 0u;
  int prev = v0 < nV ? off[v0] : 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (v0 + k >= nV) break;
    const int next = off[v0 + k + 1];
    if (next > prev) m |= 1u << k;
    prev = next;
  }
  return __popc(m);
}

__global__ void __launch_bounds__(kRThreads) k_ne_count(const int32_t *off, int nV, int32_t *part) {
  unsigned m;
  const int c = ne_flags(off, nV, blockIdx.x * kScanTile + threadIdx.x * kScanItems, m);
  int total;
  cta_scan_excl(c, &total);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kRThreads)
    k_ne_write(const int32_t *off, int nV, const int32_t *part, int32_t *vid, int32_t *end,
               int32_t *n_out) {
  unsigned m;
  const int v0 = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  const int c = ne_flags(off, nV, v0, m);
  int total;
  int pos = cta_scan_excl(c, &total) + part[blockIdx.x];
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *n_out = part[blockIdx.x] + total;
  for (; m; m &= m - 1) {
    const int v = v0 + __ffs(m) - 1;
    vid[pos] = v;
    end[pos] = off[v + 1];
    ++pos;
  }
}

// The build's temporary arrays, one allocation.
struct Scratch {
  uint8_t *base = nullptr;
  size_t used = 0;
  size_t take(size_t bytes) {
    const size_t at = used;
    used += (std::max<size_t>(bytes, 1) + 255) & ~(size_t)255;
    return at;
  }
  ~Scratch() {
    if (base) cudaFree(base);
  }
};

gas_status_t scan_excl(int32_t *a, int n, int32_t *part, cudaStream_t s) {
  if (n <= 0) return GAS_OK;
  const int nb = (int)(((long long)n + kScanTile - 1) / kScanTile);
  k_scan_reduce<<<nb, kRThreads, 0, s>>>(a, n, part);
  k_scan_spine<<<1, kRThreads, 0, s>>>(part, nb);
  k_scan_down<<<nb, kRThreads, 0, s>>>(a, n, part);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

// Stable sort of the edge indices by keys[] (values 0..n-1 enter with the
// first pass), bits >= 1.  Sorted keys end in *kres, the permutation in
// *vres (two of the four work buffers).
gas_status_t radix_sort(const int32_t *keys, int n, int bits, int32_t *k0, int32_t *v0,
                        int32_t *k1, int32_t *v1, int32_t *hist, int32_t *part,
                        int32_t **kres, int32_t **vres, cudaStream_t s) {
  const int ntiles = (int)(((long long)n + kRTile - 1) / kRTile);
  const int passes = (bits + kRBits - 1) / kRBits;
  CUDA_TRY(cudaFuncSetAttribute(k_rs_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(SortSmem)));
  const int32_t *kin = keys;
  const int32_t *vin = nullptr;
  int32_t *ko = k0, *vo = v0, *ka = k1, *va = v1;
  for (int p = 0; p < passes; ++p) {
    const int shift = kRBits * p;
    k_rs_hist<<<ntiles, kSThreads, 0, s>>>(kin, n, shift, ntiles, hist);
    GAS_TRY(scan_excl(hist, kRBins * ntiles, part, s));
    k_rs_scatter<<<ntiles, kSThreads, sizeof(SortSmem), s>>>(kin, vin, ko, vo, n, shift, ntiles,
                                                             hist);
    CUDA_TRY(cudaGetLastError());
    kin = ko;
    vin = vo;
    std::swap(ko, ka);
    std::swap(vo, va);
  }
  *kres = const_cast<int32_t *>(kin);
  *vres = const_cast<int32_t *>(vin);
  return GAS_OK;
}

}  // namespace

namespace gas {

bool device_build_for(int64_t n_edges) {
  const char *v = getenv("GAS_GRAPH_BUILD");
  if (v && strcmp(v, "host") == 0) return false;
  if (v && strcmp(v, "device") == 0) return true;
  // set_graph, host / device build: 7 K edges 0.21 / 0.24 ms sorted by source,
  // 0.21 / 0.31 unsorted; 35 K 0.57 / 0.29, 0.51 / 0.34; 1 M 18.4 / 0.6
  return n_edges >= (1 << 14);
}

gas_status_t build_graph_device(gas_engine *e, const int32_t *srcs, const int32_t *dsts,
                                const void *edge_data, std::vector<int32_t> *csc_perm,
                                std::vector<int32_t> *csr_perm, void *stream) {
  cudaStream_t s = S(stream);
  const int nV = e->nV, n = e->nE;
  const size_t eb = e->ebytes, nb = (size_t)n * 4;
  const bool have_ed = edge_data && eb > 0 && e->csc_ed;
  Scratch w;
  const size_t ntiles = (size_t)(((long long)n + kRTile - 1) / kRTile);
  const size_t hist_n = kRBins * std::max<size_t>(ntiles, 1);
  const size_t nparts = (hist_n + kScanTile - 1) / kScanTile + 1;
  const size_t at_src = w.take(nb), at_dst = w.take(nb);
  size_t at_work[4];
  for (size_t &at : at_work) at = w.take(nb);
  const size_t at_hist = w.take(hist_n * 4), at_part = w.take(nparts * 4);
  const size_t at_flags = w.take(sizeof(EdgeFlags)), at_ed = w.take(have_ed ? (size_t)n * eb : 0);
  {
    const cudaError_t ce = cudaMalloc((void **)&w.base, w.used);
    if (ce != cudaSuccess) {
      w.base = nullptr;
      cudaGetLastError();
      return fail(GAS_ERR_NOMEM, "device graph build: %s", cudaGetErrorString(ce));
    }
  }
  int32_t *src = (int32_t *)(w.base + at_src), *dst = (int32_t *)(w.base + at_dst);
  int32_t *k0 = (int32_t *)(w.base + at_work[0]), *v0 = (int32_t *)(w.base + at_work[1]);
  int32_t *k1 = (int32_t *)(w.base + at_work[2]), *v1 = (int32_t *)(w.base + at_work[3]);
  int32_t *hist = (int32_t *)(w.base + at_hist), *part = (int32_t *)(w.base + at_part);
  EdgeFlags *flags = (EdgeFlags *)(w.base + at_flags);
  uint8_t *ed = w.base + at_ed;
  if (n) {
    CUDA_TRY(cudaMemcpyAsync(src, srcs, nb, cudaMemcpyHostToDevice, s));
    CUDA_TRY(cudaMemcpyAsync(dst, dsts, nb, cudaMemcpyHostToDevice, s));
  }
  CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(EdgeFlags), s));
  const int grid = 8 * e->num_sms;
  if (n) k_check_edges<<<grid, 256, 0, s>>>(src, dst, n, nV, flags);
  if (n && have_ed)
    CUDA_TRY(cudaMemcpyAsync(ed, edge_data, (size_t)n * eb, cudaMemcpyHostToDevice, s));
  EdgeFlags f{};
  CUDA_TRY(cudaMemcpyAsync(&f, flags, sizeof(f), cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (f.bad) {
    const int i = f.bad - 1;
    return fail(GAS_ERR_INVALID, "edge %d: (%d, %d) outside [0,%d)", i, srcs[i], dsts[i], nV);
  }
  int bits = 1;
  while (bits < 31 && (1LL << bits) < nV) ++bits;  // keys are < nV <= 2^bits
  // order 0: CSC (key dst, other endpoint src); order 1: CSR (key src)
  for (int order = 0; order < 2; ++order) {
    const int32_t *key = order == 0 ? dst : src;
    const int32_t *other = order == 0 ? src : dst;
    int32_t *off = order == 0 ? e->csc_off : e->csr_off;
    int32_t *out = order == 0 ? e->csc_src : e->csr_dst;
    uint8_t *out_ed = (uint8_t *)(order == 0 ? e->csc_ed : e->csr_ed);
    std::vector<int32_t> *perm_out = order == 0 ? csc_perm : csr_perm;
    const bool sorted = !(order == 0 ? f.b_unsorted : f.a_unsorted);
    if (sorted) {  // the edge list is in this order: its own permutation
      k_offsets_from_sorted<<<grid, 256, 0, s>>>(key, n, nV, off);
      if (n) {
        CUDA_TRY(cudaMemcpyAsync(out, other, nb, cudaMemcpyDefault, s));
        if (have_ed) CUDA_TRY(cudaMemcpyAsync(out_ed, ed, (size_t)n * eb, cudaMemcpyDefault, s));
      }
      if (perm_out) {
        perm_out->resize(n);
        for (int i = 0; i < n; ++i) (*perm_out)[i] = i;
      }
    } else {
      int32_t *ks = nullptr, *vs = nullptr;
      GAS_TRY(radix_sort(key, n, bits, k0, v0, k1, v1, hist, part, &ks, &vs, s));
      k_offsets_from_sorted<<<grid, 256, 0, s>>>(ks, n, nV, off);
      k_gather_i32<<<grid, 256, 0, s>>>(other, vs, n, out);
      if (have_ed) k_gather_rec<<<grid, 256, 0, s>>>(ed, vs, n, (int)eb, out_ed);
      if (perm_out) {
        perm_out->resize(n);
        CUDA_TRY(cudaMemcpyAsync(perm_out->data(), vs, nb, cudaMemcpyDeviceToHost, s));
        CUDA_TRY(cudaStreamSynchronize(s));
      }
    }
    CUDA_TRY(cudaGetLastError());
  }
  CUDA_TRY(cudaStreamSynchronize(s));  // the work buffers are freed at return
  return GAS_OK;
}

gas_status_t device_scan_excl(int32_t *a, int n, int32_t *part, void *stream) {
  return scan_excl(a, n, part, S(stream));
}

int device_scan_parts(int n) { return (int)(((long long)n + kScanTile - 1) / kScanTile) + 1; }

gas_status_t build_ne_rows(gas_engine *e, int32_t *part, int32_t *n_out, void *stream) {
  const int nb = ne_blocks(e->nV);
  k_ne_count<<<nb, kRThreads, 0, S(stream)>>>(e->csc_off, e->nV, part);
  k_scan_spine<<<1, kRThreads, 0, S(stream)>>>(part, nb);
  k_ne_write<<<nb, kRThreads, 0, S(stream)>>>(e->csc_off, e->nV, part, e->ne_vid, e->ne_end,
                                              n_out);
  CUDA_TRY(cudaGetLastError());
  return GAS_OK;
}

int ne_blocks(int nV) { return std::max(1, (int)(((long long)nV + kScanTile - 1) / kScanTile)); }

}  // namespace gas
