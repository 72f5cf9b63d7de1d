// Multi-CTA exact top-k-by-magnitude selection and unordered compaction, shared
// by the re-selects of the two exchange kernels.  All CTAs of a rank run the same
// sequence and meet in RankBarrier.
#pragma once
#include "common.cuh"

namespace gtk {

constexpr int kSelThreads = 512;
constexpr int kStageCap = 2048;  // pairs staged in shared memory before one global cursor bump

struct SelectShared {
  unsigned int hist[kHistBins];
  unsigned int warp_tot[kSelThreads / 32];
  unsigned int res_digit;
  unsigned int res_krem;
  unsigned int res_total;
  unsigned int stage_n;
  unsigned int stage_base;
  Pair stage[kStageCap];
};

struct Threshold {
  uint32_t key;        // bit pattern of the k-th largest magnitude
  uint32_t quota;      // how many entries equal to key are still selected
  bool select_all;     // fewer live entries than k: everything is selected
  unsigned int n;      // how many entries are selected
};

__device__ __forceinline__ void smem_hist_clear(SelectShared& s) {
  for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) s.hist[i] = 0u;
  __syncthreads();
}

__device__ __forceinline__ void smem_hist_flush(SelectShared& s, unsigned int* ghist, int nbins) {
  __syncthreads();
  for (int i = threadIdx.x; i < nbins; i += kSelThreads) {
    const unsigned int c = s.hist[i];
    if (c) atomicAdd(&ghist[i], c);
  }
}

// Every CTA scans the (complete) global histogram from the top bin downwards and
// finds the digit D with count(bins > D) < k_rem <= count(bins >= D).
// Results are left in shared memory: res_digit, res_krem (k_rem minus the count
// above D), res_total (all entries).  GLOBAL: counts lies in global memory, else in this CTA's shared memory.
template <int NBINS, bool GLOBAL = true>
__device__ __forceinline__ void find_digit_in(SelectShared& s, const unsigned int* counts, unsigned int k_rem) {
  constexpr int BPT = NBINS / kSelThreads;
  static_assert(BPT >= 1, "bins per thread");
  const int t = threadIdx.x;
  unsigned int c[BPT];
  unsigned int mine = 0;
#pragma unroll
  for (int j = 0; j < BPT; ++j) {
    c[j] = GLOBAL ? __ldcg(&counts[t * BPT + j]) : counts[t * BPT + j];
    mine += c[j];
  }
  // inclusive suffix sum over threads (higher thread = higher bins)
  unsigned int suf = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int v = __shfl_down_sync(0xffffffffu, suf, o);
    if ((int)lane_id() + o < 32) suf += v;
  }
  const int w = t >> 5;
  if (lane_id() == 0) s.warp_tot[w] = suf;
  if (t == 0) { s.res_digit = 0u; s.res_krem = 0u; }
  __syncthreads();
  unsigned int above_warps = 0, total = 0;
#pragma unroll
  for (int i = 0; i < kSelThreads / 32; ++i) {
    const unsigned int v = s.warp_tot[i];
    total += v;
    if (i > w) above_warps += v;
  }
  const unsigned int above = above_warps + (suf - mine);  // entries in bins above this thread's
  if (t == 0) s.res_total = total;
  if (above < k_rem && k_rem <= above + mine) {
    unsigned int a = above;
#pragma unroll
    for (int j = BPT - 1; j >= 0; --j) {
      if (a < k_rem && k_rem <= a + c[j]) {
        s.res_digit = (unsigned int)(t * BPT + j);
        s.res_krem = k_rem - a;
      }
      a += c[j];
    }
  }
  __syncthreads();
}

// First selection level of a set whose k-th magnitude is expected (not known) at or a little above `lo`: bin 0 below lo,
// bins of 2^kBandShift keys above it (together a quarter octave), the last bin open to the top.
constexpr unsigned int kBandShift = 10u;
__device__ __forceinline__ unsigned int band_bin(uint32_t key, uint32_t lo) {
  if (key < lo) return 0u;
  const unsigned int b = 1u + ((key - lo) >> kBandShift);
  return b < (unsigned int)kHistBins ? b : (unsigned int)kHistBins - 1u;
}
constexpr unsigned int kBandList = kHistBins;  // entries of the threshold's bin that are looked at directly

// The k-th largest magnitude of the entries that visit(f) calls f(key) for, each exactly once over all CTAs.
// set: the rank's four zeroed global histogram rows for this selection, row 0 already holding the complete
// counts of band_bin(key, lo).  list_n: a zeroed global word.  As a rule one sweep and one barrier: the entries of
// the threshold's bin (a few hundred of 10^5) go into a list and every CTA counts their single keys.
// When the prediction missed (bin 0 or the last one, or too many entries), three counting sweeps over bits
// 30..20, 19..10 and 9..0.  Returns false on abort.
template <typename Visit>
__device__ __forceinline__ bool band_select_kth(SelectShared& s, RankBarrier& bar, unsigned int k, uint32_t lo,
                                                unsigned int (*set)[kHistBins], unsigned int* list_n, Visit visit,
                                                Threshold* out, uint32_t where) {
  out->key = 0u;
  out->quota = 0u;
  find_digit_in<kHistBins>(s, set[0], k);
  out->select_all = s.res_total <= k;  // not more live entries than k: keep them all
  out->n = out->select_all ? s.res_total : k;
  const unsigned int bin = s.res_digit;
  unsigned int k_rem = s.res_krem;
  __syncthreads();
  if (out->select_all) return true;
  if (bin != 0u && bin != (unsigned int)kHistBins - 1u) {
    unsigned int* const list = set[1];
    visit([&](uint32_t key) {
      if (band_bin(key, lo) != bin) return;
      const unsigned int at = atomicAdd(list_n, 1u);
      if (at < kBandList) list[at] = key;
    });
    if (!bar.sync(where)) return false;
    const unsigned int n = __ldcg(list_n);
    if (n <= kBandList) {
      constexpr uint32_t kWidth = 1u << kBandShift;
      for (unsigned int i = threadIdx.x; i < kWidth; i += kSelThreads) s.hist[i] = 0u;
      __syncthreads();
      for (unsigned int i = threadIdx.x; i < n; i += kSelThreads)
        atomicAdd(&s.hist[(__ldcg(&list[i]) - lo) & (kWidth - 1u)], 1u);
      __syncthreads();
      find_digit_in<(int)kWidth, false>(s, s.hist, k_rem);
      out->key = lo + ((bin - 1u) << kBandShift) + s.res_digit;
      out->quota = s.res_krem;
      __syncthreads();
      return true;
    }
  }
  uint32_t prefix = 0;
  k_rem = k;
  for (int pass = 0; pass < 3; ++pass) {
    unsigned int* const ghist = pass == 0 ? set[2] : set[3] + (pass == 2 ? 1024 : 0);
    const int shift = 20 - 10 * pass, nbins = pass == 0 ? kHistBins : 1024;
    smem_hist_clear(s);
    visit([&](uint32_t key) {
      if (pass == 0) atomicAdd(&s.hist[key >> 20], 1u);
      else if ((key >> (shift + 10)) == prefix) atomicAdd(&s.hist[(key >> shift) & 1023u], 1u);
    });
    smem_hist_flush(s, ghist, nbins);
    if (!bar.sync(where + 1 + pass)) return false;
    if (pass == 0) find_digit_in<kHistBins>(s, ghist, k_rem);
    else find_digit_in<1024>(s, ghist, k_rem);
    prefix = pass == 0 ? s.res_digit : (prefix << 10) | s.res_digit;
    k_rem = s.res_krem;
    __syncthreads();
  }
  out->key = prefix;
  out->quota = k_rem;
  return true;
}

// CTA-wide staged append.  Call put() from any thread, at most once, then end_tile(whether it has) from all threads,
// once per loop trip; place(pair, position) stores an entry.  Whether the stage is full is decided from a count that every
// thread of the CTA gets from the barrier: read from shared memory behind it, a fast thread's next put() could
// reach a slow one's look at the counter, which then flushed alone.
struct StagedAppender {
  SelectShared* s;
  unsigned int* cursor;  // global cursor (local memory)
  unsigned int cap;
  Ctrl* ctrl;
  unsigned int staged;   // the same in all threads

  __device__ __forceinline__ void begin() {
    staged = 0u;
    if (threadIdx.x == 0) s->stage_n = 0u;
    __syncthreads();
  }
  __device__ __forceinline__ void put(Pair p) {
    const unsigned int pos = atomicAdd(&s->stage_n, 1u);
    s->stage[pos] = p;
  }
  template <typename Place>
  __device__ __forceinline__ void flush(Place place) {
    if (staged == 0u) return;
    if (threadIdx.x == 0) {
      s->stage_base = atomicAdd(cursor, staged);
      s->stage_n = 0u;
    }
    __syncthreads();
    const unsigned int base = s->stage_base;
    for (unsigned int i = threadIdx.x; i < staged; i += kSelThreads) {
      const unsigned int pos = base + i;
      if (pos < cap) place(s->stage[i], pos);
      else record_error(ctrl, ST_CAPACITY, 900);
    }
    staged = 0u;
    __syncthreads();
  }
  template <typename Place>
  __device__ __forceinline__ void end_tile(bool has_put, Place place) {
    staged += (unsigned int)__syncthreads_count(has_put);
    if (staged > (unsigned int)(kStageCap - kSelThreads)) flush(place);
  }
};

// Decide one entry against the threshold.  Entries equal to the threshold take a
// ticket; the first `quota` tickets are selected.
__device__ __forceinline__ bool passes_threshold(uint32_t key, const Threshold& th,
                                                 unsigned int* tie_counter) {
  if (th.select_all) return true;
  if (key > th.key) return true;
  if (key == th.key) return atomicAdd(tie_counter, 1u) < th.quota;
  return false;
}

}  // namespace gtk
