// gas_grid.cuh -- helpers of the persistent cooperative kernels (the small-
// graph BFS, the push tail): a grid barrier whose wait is bounded, and warp-
// aggregated counters.  Not installed.
#ifndef GAS_GRID_CUH_
#define GAS_GRID_CUH_

#include <cuda_runtime.h>

namespace gasgrid {

// polls of about 0.6 us: a wait gives up after some seconds
constexpr long long kMaxSpins = 1LL << 23;

// The barrier's state: zeroed once, and again after a launch that failed.
// Three arrival words in rotation: barrier i counts in word i % 3, and once
// it is passed nobody polls word (i - 1) % 3 any more, which is cleared then
// and next used by barrier i + 2.  So no CTA resets what others poll, and
// there is no second round trip to release the waiters: an arrival is one
// reduction, a wait polls the same word (measured with 28 to 152 CTAs: about
// 3,700 cycles with the control value's load, against 5,800 with a count, its
// reset and a generation word; BFS on R-MAT 2^16 136 -> 108 us).
// next: the word the following launch begins with.
struct Barrier {
  unsigned int word[3];
  unsigned int next;
};
constexpr unsigned int kGaveUp = 1u << 30;

// Every CTA of a cooperative launch calls it; index (0..2, thread 0's copy
// counts) starts at next and goes back there at the end.  Returns false in all
// threads when a wait gave up (here or in another CTA), and the caller leaves
// the kernel.  with(): run by thread
// 0 after the wait, its result returned in *out to every thread of the CTA
// (one load for the CTA instead of one per thread).
template <class T, class F>
__device__ __forceinline__ bool barrier_with(Barrier *b, unsigned int &index, T *out, F with) {
  __shared__ T s_out;
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int *w = &b->word[index];
    __threadfence();
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(w) : "memory");
    unsigned int seen = 0;
    long long spins = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(w) : "memory");
      if (seen >= gridDim.x) break;
      if (++spins > kMaxSpins) {
        atomicAdd(w, kGaveUp);
        seen = kGaveUp;
        break;
      }
      if (spins > 64) __nanosleep(64);
    }
    __threadfence();
    s_ok = seen < kGaveUp;
    if (blockIdx.x == 0) b->word[index ? index - 1u : 2u] = 0u;
    index = index == 2u ? 0u : index + 1u;
    s_out = with();
  }
  __syncthreads();
  *out = s_out;
  return s_ok != 0;
}

// The same among the CTAs of one cluster that is the whole grid: the hardware's
// barrier, which orders global memory within the cluster and cannot give up.
// Runs of small graphs take half a microsecond to a microsecond less per
// barrier: BFS on R-MAT 1 K, 4 K and 16 K vertices 68 -> 59, 57 and 60 us,
// SSSP on R-MAT 2 K 112 -> 105, Erdos-Renyi 2 K 119 -> 106.
template <class T, class F>
__device__ __forceinline__ void cluster_barrier_with(T *out, F with) {
  __shared__ T s_out;
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (threadIdx.x == 0) s_out = with();
  __syncthreads();
  *out = s_out;
}

__device__ __forceinline__ long long warp_sum(long long v) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

__device__ __forceinline__ int warp_incl_sum(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += o;
  }
  return v;
}

// Adds a per-thread count to *dst, one atomic per warp (all lanes call).
__device__ __forceinline__ void warp_add(long long v, long long *dst) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0 && v)
    atomicAdd((unsigned long long *)dst, (unsigned long long)v);
}

}  // namespace gasgrid

#endif  // GAS_GRID_CUH_
