// Exact selection of the k-th largest magnitude in wide CTAs (1024 threads, one
// or a cluster of them): levels of 2048 bins over the range of keys that still
// matters, and ordered placement of what was selected.  Shared by k1_pick and the
// table form of the tree exchange.
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"

namespace gtk {

constexpr int kPickThreads = 1024;
constexpr int kBins = kHistBins;           // 2048: two per thread

struct WideShared {
  unsigned int hist[kBins];
  unsigned int warp_tot[kPickThreads / 32];
  unsigned int warp_n[2][kPickThreads / 32];
  unsigned int base[2];
  unsigned int res_bin, res_krem, res_n;
};

// The keys that still matter: lo <= key <= hi, in bins of 2^shift.  An open level clamps everything
// above its last bin into it.
struct Level {
  uint32_t lo, hi;
  unsigned int shift;
  bool open;
  __device__ __forceinline__ bool has(uint32_t key) const { return key - lo <= hi - lo; }
  __device__ __forceinline__ unsigned int bin(uint32_t key) const {
    const unsigned int b = (key - lo) >> shift;
    return b < (unsigned int)kBins ? b : (unsigned int)kBins - 1u;
  }
  // The level inside bin b; false when the bin is a single key (then lo is that key).
  __device__ __forceinline__ bool narrow(unsigned int b) {
    lo += b << shift;
    if (!(open && b == (unsigned int)kBins - 1u)) {
      if (shift == 0u) return false;
      hi = lo + ((1u << shift) - 1u);
    }
    const uint32_t width = hi - lo;  // an open top is as wide as the keys go
    const int bits = 32 - __clz(width);
    shift = bits > 11 ? (unsigned int)(bits - 11) : 0u;
    open = false;
    return true;
  }
};

// Finds the bin B with count(bins > B) < k_rem <= count(bins >= B): res_bin, and k_rem minus the count
// above it: res_krem, and its own count: res_n.  c: the complete counts of bins 2t and 2t + 1.  Returns the sum of all counts; when it
// is below k_rem there is no such bin and the results are not set.
__device__ __forceinline__ unsigned int find_bin(WideShared& s, uint2 c, unsigned int k_rem) {
  const int t = threadIdx.x, w = t >> 5;
  const unsigned int mine = c.x + c.y;
  unsigned int suf = mine;  // inclusive suffix sum over the warp (higher lane = higher bins)
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int v = __shfl_down_sync(0xffffffffu, suf, o);
    if ((int)lane_id() + o < 32) suf += v;
  }
  if (lane_id() == 0) s.warp_tot[w] = suf;
  __syncthreads();
  const unsigned int v = s.warp_tot[lane_id()];
  const unsigned int above = __reduce_add_sync(0xffffffffu, (int)lane_id() > w ? v : 0u) + (suf - mine);
  if (above < k_rem && k_rem <= above + mine) {
    const bool upper = k_rem <= above + c.y;
    s.res_bin = 2u * t + (upper ? 1u : 0u);
    s.res_krem = k_rem - above - (upper ? 0u : c.y);
    s.res_n = upper ? c.y : c.x;
  }
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, v);
}

// Output position of the first of this thread's n entries.  cursor: global list cursor, or nullptr when
// this CTA writes the whole list.  turn alternates between consecutive calls.
__device__ __forceinline__ unsigned int place(WideShared& s, unsigned int n, unsigned int* cursor, unsigned int turn) {
  const int w = threadIdx.x >> 5;
  unsigned int pre = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int v = __shfl_up_sync(0xffffffffu, pre, o);
    if ((int)lane_id() >= o) pre += v;
  }
  if (lane_id() == 31) s.warp_n[turn & 1u][w] = pre;
  __syncthreads();
  const unsigned int v = s.warp_n[turn & 1u][lane_id()];
  const unsigned int before = __reduce_add_sync(0xffffffffu, (int)lane_id() < w ? v : 0u);
  unsigned int base = 0;
  if (cursor) {
    const unsigned int total = __reduce_add_sync(0xffffffffu, v);
    if (threadIdx.x == 0) s.base[turn & 1u] = total ? atomicAdd(cursor, total) : 0u;
    __syncthreads();
    base = s.base[turn & 1u];
  }
  return base + before + pre - n;
}

// The same for a warp's n entries: the position of the first.  cursor: not nullptr.
__device__ __forceinline__ unsigned int place_warp(WideShared& s, unsigned int n, unsigned int* cursor, unsigned int turn) {
  const int w = threadIdx.x >> 5;
  if (lane_id() == 0) s.warp_n[turn & 1u][w] = n;
  __syncthreads();
  const unsigned int v = s.warp_n[turn & 1u][lane_id()];
  const unsigned int before = __reduce_add_sync(0xffffffffu, (int)lane_id() < w ? v : 0u);
  const unsigned int total = __reduce_add_sync(0xffffffffu, v);
  if (threadIdx.x == 0) s.base[turn & 1u] = total ? atomicAdd(cursor, total) : 0u;
  __syncthreads();
  return s.base[turn & 1u] + before;
}

// One entry against the threshold; called by whole warps.  Entries equal to it take tickets, the first
// `quota` of which are selected.
__device__ __forceinline__ bool passes(bool live, uint32_t key, uint32_t th, unsigned int quota, unsigned int* tie) {
  const bool equal = live && key == th;
  bool win = live && key > th;
  const unsigned int m = __ballot_sync(0xffffffffu, equal);
  if (m) {
    unsigned int base = 0;
    if (lane_id() == (unsigned int)(__ffs(m) - 1)) base = atomicAdd(tie, (unsigned int)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    if (equal) win = base + __popc(m & lanemask_lt()) < quota;
  }
  return win;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace gtk
