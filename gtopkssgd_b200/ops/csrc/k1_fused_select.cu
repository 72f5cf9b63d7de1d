// K1: fused residual add + magnitude top-k selection + residual write-back, two
// kernels behind one call.
//
// Replaces the op sequence of the reference's TopKCompressor.compress
// (compression.py:32-57: add_, abs, topk, gather, mask fill/scatter, mul, sub_)
// and the gather of the selected values (allreducer.py:543).
//
// k1_stream  one pass over g and r (read 8d bytes, write 4d):
//     acc = g*scale + r; entries with |acc| >= tau become candidates (appended to
//     a bounded list, r <- 0), all others r <- acc.  tau is a device-resident
//     prediction from the previous call.
//     Non-finite entries (+-Inf, NaN) count as the largest magnitudes on both paths,
//     NaN above Inf, as torch.topk(|acc|) ranks them: they are selected, never left
//     in the residual.
// k1_pick    normal mode (k <= C <= cap candidates): finds the k-th magnitude
//     among the candidates, compacts the k winners, returns the rejected
//     candidates to r and re-predicts tau from the measured tail slope.
//     exact mode (C < k or the list overflowed; always on the first call, when
//     tau is +inf): restores r = acc from the stored candidates, then runs a
//     3-pass radix select over all d entries of r and one collect pass.
// The output is k (int32 index, fp32 value) pairs in no particular order.  The dense
// sparsified gradient of the reference is not materialised, except by gtk_k1_compress,
// where the stream pass leaves zeros in g and k1_pick puts the winners back, next to
// their int64 indices and values as separate lists.
//
// Why two kernels: as one cooperative kernel the two halves met in a grid barrier
// (1.3 us plus the wait for the slowest CTA), and a cooperative launch cannot
// overlap with its predecessor (launch.cuh).  The boundary between the two costs
// about as much as the barrier did, and both now start in the shadow of the
// kernel before them.
//
// No CTA waits for one that may not have started: within k1_pick, work that others
// wait for is handed out by tickets, and a CTA only waits for tickets that running
// CTAs hold; fixed shares are for work that nobody waits for.  So no co-residency is
// needed, whatever else runs on the device.
//
// No host-side clearing: the caller provides two control blocks; call i uses
// block (i & 1) and the stream pass zeroes the other one for call i + 1 (i is
// K1State::n_calls, read on the device, so the launches can be replayed from a
// CUDA graph).  k1_stream reads only n_calls and k1_pick only stream_calls, each
// written by the other kernel, so a late CTA never sees its call's own update.
#include <atomic>
#include <cstddef>
#include <type_traits>
#include "pick_common.cuh"
#include "host_api.h"
#include "launch.cuh"

namespace gtk {

constexpr int kK1Threads = 512;            // k1_stream
constexpr int kWarpStage = 128;            // pairs staged per warp
constexpr int kWarpFlushAt = kWarpStage - 32;
// From this many float4 per array on (20 M elements) the stream pass hands work out dynamically; below it the
// static split is as fast or faster (whole call: 59.0 against 60.3 us at 25.6 M, but 30.6 against 30.0 at 14.7 M).
constexpr long long kDynamicMinVec = 5ll * 1000 * 1000;
constexpr unsigned int kShards = 16;       // ticket counters of the dynamic stream pass
// Up to kPickSmall candidates one CTA selects among them, up to kPickCluster one cluster of 8 CTAs, both from
// registers; above, and in a launch without clusters (gtk_k1_pick_is_wide), all CTAs share them out.  At the borders: one CTA 2.9 us at 2.6 K candidates and 2 us more
// than the cluster at 10 K; the cluster against the shares 31.85 and 31.3 us (select + update of 8 M at 0.003, 31 K
// candidates, the cluster in launches that have one) or 1 us less than them (2.5 M at 0.01).
constexpr unsigned int kPickSmall = 4096;
constexpr unsigned int kPickCluster = 32768;
constexpr int kPickCtas = 8;               // CTAs per cluster
// The first level is counted in the stream pass from here on: see k1_launch_with.
constexpr unsigned int kCountFrom = kPickCluster / 8 * 3;

// Bins of the first selection level: (key - lo) >> shift, the last bin open to the top.  lo is the candidate
// threshold and shift puts the previous call's k-th magnitude into bins 256..511, so that the new one lies in
// a bin of its own width even when the tail is steep (bits of the key itself would put almost all candidates
// into two or three bins, whose counters then serialise the whole CTA).
struct Bands {
  uint32_t lo;
  unsigned int shift;
  __device__ __forceinline__ unsigned int bin(uint32_t key) const {  // key >= lo
    const unsigned int b = (key - lo) >> shift;
    return b < (unsigned int)kBins ? b : (unsigned int)kBins - 1u;
  }
};
__device__ __forceinline__ Bands first_bands(float tau, float kth) {
  const uint32_t lo = mag_key(tau), hi = mag_key(kth);
  const uint32_t w = hi > lo ? hi - lo : 1u;
  const int top = 31 - __clz(w);
  return Bands{lo, top > 8 ? (unsigned int)(top - 8) : 0u};
}

struct StreamShared {
  Pair wstage[kK1Threads / 32][kWarpStage];  // per-warp candidate staging
  unsigned int warp_n[kK1Threads / 32];
  unsigned int base;
  unsigned int hist[kBins];                  // this CTA's candidates (counted only when k is large)
};
// bytes of a control block that K1 dirties: header, trace, three rows of one histogram set
// (candidate levels in set 0, exact mode in set 1)
constexpr size_t kK1ClearBytes = offsetof(Ctrl, hist) + 2 * sizeof(((Ctrl*)0)->hist[0]);

// The warp's staged candidates to list positions base...; what does not fit stays in the residual.
__device__ __forceinline__ void warp_store(const Pair* wbuf, unsigned int n, unsigned int base, Pair* cand,
                                           unsigned int cap, float* r) {
  for (unsigned int i = lane_id(); i < n; i += 32) {
    const Pair p = wbuf[i];
    if (base + i < cap) st_pair(&cand[base + i], p);
    else r[p.idx] = p.val;
  }
}
__device__ __forceinline__ void warp_flush(Pair* wbuf, unsigned int& wcnt, Pair* cand, unsigned int cap,
                                           unsigned int* counter, float* r) {
  __syncwarp();
  unsigned int base = 0;
  if (lane_id() == 0) base = atomicAdd(counter, wcnt);
  base = __shfl_sync(0xffffffffu, base, 0);
  warp_store(wbuf, wcnt, base, cand, cap, r);
  wcnt = 0;
  __syncwarp();
}

// Where the gradient of a float4 position comes from: one vector, or one tensor per parameter.
struct FlatGrad {
  float* g;        // behind the scalar head
  __device__ __forceinline__ unsigned int find(long long) const { return 0u; }
  __device__ __forceinline__ float4 vec(long long v, unsigned int) const {
    return __ldcs(reinterpret_cast<const float4*>(g) + v);
  }
};
// Segment s covers the float4 positions start[s] <= v < start[s + 1] of the flat layout (parameters begin at
// multiples of four elements) and holds len[s] elements; g[s] is its gradient, nullptr for a parameter that got
// none.  A warp looks its row of 32 positions up with two ballots over the starts in shared memory (at most 1024; a
// binary search per thread made the pass over VGG-16's 54 tensors 9 us longer than over one vector), and a row that
// lies inside one aligned segment, which is nearly every one, is then read like a plain vector.
template <int N>
struct GradPointers {
  const float* g[N];
};
struct SegmentedGrad {
  const float* const* g;       // kernel parameters
  const unsigned int* start;   // shared memory, n + 1 words
  const unsigned int* len;     // shared memory
  unsigned int n;
  // The segment of the first position of v's row; all lanes of a warp, in the same row.
  __device__ __forceinline__ unsigned int find(long long v) const {
    const unsigned int row = (unsigned int)v & ~31u;
    unsigned int first = 0u;
    if (n > 32u) first = 32u * (__popc(__ballot_sync(0xffffffffu, 32u * lane_id() < n && start[32u * lane_id()] <= row)) - 1u);
    const unsigned int i = first + lane_id();
    return first + __popc(__ballot_sync(0xffffffffu, i < n && start[i] <= row)) - 1u;
  }
  // The gradient at position v of the row whose first segment is lo.
  __device__ __forceinline__ float4 vec(long long v64, unsigned int lo) const {
    const unsigned int v = (unsigned int)v64, end = (v | 31u) + 1u;
    if (end <= start[lo + 1u] && (end - start[lo]) * 4u <= len[lo] && (reinterpret_cast<uintptr_t>(g[lo]) & 15u) == 0u) {
      if (g[lo] == nullptr) return make_float4(0.f, 0.f, 0.f, 0.f);
      return __ldcs(reinterpret_cast<const float4*>(g[lo]) + (v - start[lo]));
    }
    while (v >= start[lo + 1u]) ++lo;
    const float* src = g[lo];
    const unsigned int at = (v - start[lo]) * 4u, left = len[lo] - min(at, len[lo]);
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (src == nullptr) return x;
    src += at;
    if (left >= 4u && (reinterpret_cast<uintptr_t>(src) & 15u) == 0u) return __ldcs(reinterpret_cast<const float4*>(src));
    if (left > 0u) x.x = __ldcs(src);
    if (left > 1u) x.y = __ldcs(src + 1);
    if (left > 2u) x.z = __ldcs(src + 2);
    if (left > 3u) x.w = __ldcs(src + 3);
    return x;
  }
};

// What a thread of the stream pass carries along.
struct StreamCtx {
  float* r;
  Pair* cand;
  unsigned int cap;
  unsigned int* counter;
  float scale;
  uint32_t tau_key;
  Bands bands;
  Pair* wbuf;
  unsigned int wcnt;
};

// Appends the lanes' candidates (warp-uniform call).
template <bool HIST>
__device__ __forceinline__ void take_candidates(StreamShared& ss, StreamCtx& c, bool is, long long idx, float a) {
  const unsigned int m = __ballot_sync(0xffffffffu, is);
  if (!m) return;
  if (is) {
    Pair p;
    p.idx = (int32_t)idx;
    p.val = a;
    c.wbuf[c.wcnt + __popc(m & lanemask_lt())] = p;
    if (HIST) atomicAdd(&ss.hist[c.bands.bin(mag_key(a))], 1u);
  }
  c.wcnt += __popc(m);
  if (c.wcnt > (unsigned int)kWarpFlushAt) warp_flush(c.wbuf, c.wcnt, c.cand, c.cap, c.counter, c.r);
}

// One tile of the stream pass: U float4 of g and of r per thread, STRIDE
// float4 apart (the CTA's 512 threads or one warp's 32 lanes work side by side).
template <int STRIDE, int U, bool HIST, bool ZERO, typename G>
__device__ __forceinline__ void stream_tile(long long v0, long long nvec, long long head, const G& g, float4* r4,
                                            StreamShared& ss, StreamCtx& c) {
  // Candidates are decided on the bit pattern of |acc|, which orders like the magnitude for finite
  // values and puts +-Inf and NaN on top: a non-finite entry is a candidate on this path exactly as it
  // is the largest key on the exact path (torch.topk(|acc|) in compression.py:43 also ranks NaN first).
  float4 gv[U], rv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long v = v0 + (long long)u * STRIDE;
    rv[u] = v < nvec ? r4[v] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long v = v0 + (long long)u * STRIDE;
    const unsigned int at = g.find(v);
    gv[u] = v < nvec ? g.vec(v, at) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long v = v0 + (long long)u * STRIDE;
    const bool inb = v < nvec;
    float a[4];
    a[0] = fmaf(gv[u].x, c.scale, rv[u].x);
    a[1] = fmaf(gv[u].y, c.scale, rv[u].y);
    a[2] = fmaf(gv[u].z, c.scale, rv[u].z);
    a[3] = fmaf(gv[u].w, c.scale, rv[u].w);
    bool is[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) is[e] = inb && (mag_key(a[e]) >= c.tau_key);
    if (inb) {
      float4 o;
      o.x = is[0] ? 0.f : a[0];
      o.y = is[1] ? 0.f : a[1];
      o.z = is[2] ? 0.f : a[2];
      o.w = is[3] ? 0.f : a[3];
      r4[v] = o;
      if constexpr (ZERO) reinterpret_cast<float4*>(g.g)[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (__any_sync(0xffffffffu, is[0] | is[1] | is[2] | is[3])) {
#pragma unroll
      for (int e = 0; e < 4; ++e) take_candidates<HIST>(ss, c, is[e], head + (v << 2) + e, a[e]);
    }
  }
}

// ZERO: g <- 0 on the way (a constant in a template, so that the training path has no store to g).
// G: FlatGrad (its pointer still at the vector's beginning) or SegmentedGrad (r 16-byte aligned).
template <bool HIST, bool DYNAMIC, bool ZERO, typename G>
__device__ __forceinline__ void stream_pass(StreamShared& ss, G g, float* r, const float* g_scale, long long d, Pair* cand,
                                            unsigned int cap, K1State* st, Ctrl* ctrl_pair) {
  constexpr bool kFlat = std::is_same_v<G, FlatGrad>;
  constexpr int U = DYNAMIC ? 4 : 2;  // float4 loads of g and of r in flight per thread
  const unsigned int calls = st->n_calls;
  const float tau = st->tau;
  Ctrl* ctrl = ctrl_pair + (calls & 1u);
  if (blockIdx.x == 0 && threadIdx.x == 0) st->stream_calls = calls + 1u;
  trace_stamp(ctrl, 0);
  StreamCtx c;
  c.r = r;
  c.cand = cand;
  c.cap = cap;
  c.counter = &ctrl->n_out;
  c.scale = g_scale ? *g_scale : 1.0f;
  c.tau_key = __float_as_uint(tau);
  c.bands = first_bands(tau, st->kth_mag);
  c.wbuf = ss.wstage[threadIdx.x >> 5];
  c.wcnt = 0;
  if (HIST) __syncthreads();

  // Leading scalars up to the first 16-byte boundary (g and r share the offset).
  const unsigned int mis = (unsigned int)((reinterpret_cast<uintptr_t>(r) >> 2) & 3u);
  long long head = mis ? (4 - mis) : 0;
  if (head > d) head = d;
  const long long nvec = (d - head) >> 2;
  const long long tail0 = head + (nvec << 2);
  if constexpr (kFlat) g.g += head;
  float4* r4 = reinterpret_cast<float4*>(r + head);

  if (!DYNAMIC) {
    // Static split: CTA b takes tiles b, b + grid, ...; every load instruction of the CTA covers 8 KB.
    // (One contiguous, equally sized range per CTA was tried: its ragged last tile costs almost a full
    // tile's latency in every CTA, and the call got 3 % slower at d = 25.6 M.)
    constexpr long long kTileVec = (long long)kK1Threads * U;
    const long long ntiles = (nvec + kTileVec - 1) / kTileVec;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
      stream_tile<kK1Threads, U, HIST, ZERO>(tile * kTileVec + threadIdx.x, nvec, head, g, r4, ss, c);
  } else {
    // Large vectors: SMs do not all see the same memory bandwidth, and with the static split the slowest
    // CTA ended up to 13 us (d = 64 M) after the first.  Here work is handed out per warp in tiles of 32 lanes
    // x U float4: the first tile of a warp is fixed, further ones come from a ticket counter that is read one
    // tile ahead, so the atomic's latency hides behind the loads.  kShards counters, each for every kShards-th
    // warp and tile: one counter cannot serve a ticket per ns, and longer chunks (four tiles, 17 us each at
    // the end) let the last warp finish 8 us after the first.
    constexpr long long kWarpTileVec = 32ll * U;
    const long long ntiles = (nvec + kWarpTileVec - 1) / kWarpTileVec;
    const unsigned int warp = blockIdx.x * (kK1Threads / 32) + (threadIdx.x >> 5);
    const unsigned int shard = warp % kShards;
    const unsigned int warps = (gridDim.x * (kK1Threads / 32) - shard + kShards - 1u) / kShards;  // of this shard
    unsigned int* ticket = &ctrl->hist[1][3][shard * 32u];  // 128 bytes apart; this row is not used otherwise
    long long turn = warp / kShards;
    for (long long tile = warp; tile < ntiles; tile = turn * kShards + shard) {
      unsigned int nxt = 0;
      if (lane_id() == 0) nxt = atomicAdd(ticket, 1u);  // consumed after this tile
      stream_tile<32, U, HIST, ZERO>(tile * kWarpTileVec + lane_id(), nvec, head, g, r4, ss, c);
      turn = (long long)warps + __shfl_sync(0xffffffffu, nxt, 0);
    }
  }
  // Scalar head and tail (at most 3 + 3 entries), one warp of CTA 0.
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    const long long nscalar = head + (d - tail0);
    bool is = false;
    float a = 0.f;
    long long i = 0;
    const long long j = lane_id();
    const unsigned int last = g.find(nvec);  // the row of the tail
    if (j < nscalar) {
      i = j < head ? j : tail0 + (j - head);
      float gi;
      if constexpr (kFlat) {
        gi = g.g[i - head];
      } else {  // (head is 0) the last float4 position, of which only some elements exist
        const float4 x = g.vec(i >> 2, last);
        gi = (i & 3) == 0 ? x.x : (i & 3) == 1 ? x.y : x.z;
      }
      a = fmaf(gi, c.scale, r[i]);
      is = mag_key(a) >= c.tau_key;
      r[i] = is ? 0.f : a;
      if constexpr (ZERO) g.g[i - head] = 0.f;
    }
    take_candidates<HIST>(ss, c, is, i, a);
  }
  // The other control block, for the next call (its last user ended before this kernel began).
  {
    uint4* other = reinterpret_cast<uint4*>(ctrl_pair + ((calls & 1u) ^ 1u));
    const size_t nvec16 = kK1ClearBytes / 16;
    for (size_t i = (size_t)blockIdx.x * kK1Threads + threadIdx.x; i < nvec16; i += (size_t)gridDim.x * kK1Threads)
      other[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  // One list reservation for what the CTA's warps still hold: a reservation per warp queues thousands of
  // atomics on one address just when all CTAs finish.
  const int w = threadIdx.x >> 5;
  if (lane_id() == 0) ss.warp_n[w] = c.wcnt;
  __syncthreads();
  unsigned int before = 0, total = 0;
#pragma unroll
  for (int q = 0; q < kK1Threads / 32; ++q) {
    const unsigned int n = ss.warp_n[q];
    if (q < w) before += n;
    total += n;
  }
  if (total) {
    if (threadIdx.x == 0) ss.base = atomicAdd(c.counter, total);
    __syncthreads();
    warp_store(c.wbuf, c.wcnt, ss.base + before, cand, cap, r);
  }
  if (HIST) {  // publish this CTA's part of the first level
    for (int i = threadIdx.x; i < kBins; i += kK1Threads) {
      const unsigned int n = ss.hist[i];
      if (n) atomicAdd(&ctrl->hist[0][0][i], n);
    }
  }
  trace_stamp(ctrl, 1);  // CTA 0 finished its share
}

template <bool HIST, bool DYNAMIC, bool ZERO>
__global__ void __launch_bounds__(kK1Threads, 2)
k1_stream(float* g, float* r, const float* g_scale, long long d, Pair* cand, unsigned int cap, K1State* st,
          Ctrl* ctrl_pair) {
  __shared__ StreamShared ss;
  if (HIST)
    for (int i = threadIdx.x; i < kBins; i += kK1Threads) ss.hist[i] = 0u;
  pdl_begin(g, r, g_scale, st, ctrl_pair);
  stream_pass<HIST, DYNAMIC, ZERO>(ss, FlatGrad{g}, r, g_scale, d, cand, cap, st, ctrl_pair);
}

// segments: n + 1 start positions, then n lengths.
template <bool HIST, bool DYNAMIC, int N>
__global__ void __launch_bounds__(kK1Threads, 2)
k1_stream_segments(const __grid_constant__ GradPointers<N> g, const unsigned int* segments, unsigned int n, float* r,
                   long long d, Pair* cand, unsigned int cap, K1State* st, Ctrl* ctrl_pair) {
  __shared__ StreamShared ss;
  __shared__ unsigned int seg[2 * N + 1];
  if (HIST)
    for (int i = threadIdx.x; i < kBins; i += kK1Threads) ss.hist[i] = 0u;
  pdl_begin(segments, r, st, ctrl_pair);
  for (unsigned int i = threadIdx.x; i < 2u * n + 1u; i += kK1Threads) seg[i] = segments[i];
  __syncthreads();
  const float* no_scale = nullptr;
  stream_pass<HIST, DYNAMIC, false>(ss, SegmentedGrad{g.g, seg, seg + n + 1, n}, r, no_scale, d, cand, cap, st, ctrl_pair);
}

// ---------------------------------------------------------------------------
// k1_pick
// ---------------------------------------------------------------------------
// Where a winner goes: the pair list, and for gtk_k1_compress the other forms.
struct Winners {
  Pair* sel;
  float* dense;        // nullptr: pairs only
  long long* idx;
  float* val;
  __device__ __forceinline__ Winners from(unsigned int pos) const {
    return Winners{sel + pos, dense, idx ? idx + pos : nullptr, val ? val + pos : nullptr};
  }
  __device__ __forceinline__ void put(unsigned int pos, Pair e) const {
    st_pair(&sel[pos], e);
    if (dense) {
      dense[e.idx] = e.val;
      idx[pos] = e.idx;
      val[pos] = e.val;
    }
  }
};

constexpr unsigned int kAside = 256;  // entries of the threshold's bin that one thread each ranks
struct PickShared : WideShared {
  unsigned int share[3][kBins / kPickCtas]; // cluster: the sums of bins b = rank (mod 8), a buffer per level in turn
  unsigned int chunk;
  unsigned int tie;
  unsigned int cta_n[kPickCtas];
  int ok;
  // Entries of the threshold's bin (one CTA, cluster: in CTA 0), their keys apart for the ranking.
  __align__(16) uint32_t aside_key[kAside];
  Pair aside[kAside];
  unsigned int aside_n;
  uint32_t kth;
};

__device__ __forceinline__ uint2 global_counts(const unsigned int* ghist) {
  return __ldcg(reinterpret_cast<const uint2*>(ghist) + threadIdx.x);
}
__device__ __forceinline__ uint2* my_bins(PickShared& s) {
  return reinterpret_cast<uint2*>(s.hist) + threadIdx.x;
}
__device__ __forceinline__ void publish_hist(PickShared& s, unsigned int* ghist) {
  const uint2 c = *my_bins(s);
  if (c.x) atomicAdd(&ghist[2 * threadIdx.x], c.x);
  if (c.y) atomicAdd(&ghist[2 * threadIdx.x + 1], c.y);
}

// Calls f(chunk) for every chunk this CTA gets of phase ph; returns how many.
template <typename F>
__device__ __forceinline__ unsigned int for_chunks(PickShared& s, Ctrl* ctrl, int ph, unsigned int nchunks, F f) {
  unsigned int mine = 0, next = 0;
  if (threadIdx.x == 0) next = atomicAdd(&ctrl->ticket[ph], 1u);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s.chunk = next;
    __syncthreads();
    const unsigned int chunk = s.chunk;
    if (chunk >= nchunks) return mine;
    if (threadIdx.x == 0) next = atomicAdd(&ctrl->ticket[ph], 1u);  // arrives while this chunk is worked on
    f(chunk);
    ++mine;
  }
}
// Reports this CTA's chunks of phase ph as done (all threads' work before it included); true in thread 0
// of the CTA that completes the phase.
__device__ __forceinline__ bool report(Ctrl* ctrl, int ph, unsigned int mine, unsigned int nchunks) {
  __syncthreads();
  if (threadIdx.x != 0 || mine == 0u) return false;
  __threadfence();
  return atomicAdd(&ctrl->done[ph], mine) + mine == nchunks;
}
// Waits until the phase is complete.  All its tickets are taken by running CTAs when a CTA gets here.
__device__ __forceinline__ bool wait_phase(PickShared& s, Ctrl* ctrl, int ph, unsigned int nchunks,
                                           uint64_t limit_ns, uint32_t where) {
  if (threadIdx.x == 0) {
    int ok = 1;
    const uint64_t t0 = globaltimer_ns();
    unsigned int spins = 0;
    while (ld_acquire_gpu_u32(&ctrl->done[ph]) < nchunks) {
      if (aborted(ctrl)) { ok = 0; break; }
      if ((++spins & 63u) == 0u && globaltimer_ns() - t0 > limit_ns) {
        record_error(ctrl, ST_TIMEOUT_BARRIER, where);
        ok = 0;
        break;
      }
    }
    s.ok = ok;
  }
  __syncthreads();
  return s.ok != 0;
}

// State for the next call: tau such that its stream pass finds about ratio * k candidates, from a
// power-law tail count(t) = k * (t / t_k)^(-alpha) whose exponent is measured from (C candidates at the tau
// used, k entries at t_k) and smoothed.  Every candidate beyond k costs an append, a count and a scattered
// write back, a shortfall costs an exact pass.  So ratio adapts to how well the predictions have
// hit lately (|log(found / aimed)|, decaying maximum) and to the sampling noise of a small k, at most
// target_ratio.
// `was` is the state as the kernel found it.
__device__ __forceinline__ void finish_state(K1State* st, const K1State& was, uint32_t key_k, unsigned int n_sel,
                                             unsigned int k, unsigned int count, unsigned int C, bool exact,
                                             float target_ratio) {
  const float t_k = __uint_as_float(key_k), tau = was.tau;
  float alpha = was.alpha, slack = was.slack;
  const unsigned int aimed = was.aimed;
  const float ratio_found = (float)C / (float)k;
  if (!exact && tau > 0.f && tau < t_k * 0.9999f && ratio_found > 1.02f && isfinite(t_k)) {
    float m = logf(ratio_found) / logf(t_k / tau);
    m = fminf(fmaxf(m, 2.0f), 1024.0f);
    alpha = alpha > 0.f ? 0.5f * (alpha + m) : m;
  }
  slack *= 0.9f;
  if (exact) {
    slack = 1.f;
  } else if (aimed) {
    slack = fmaxf(slack, fabsf(logf((float)C / (float)aimed)));
  }
  const float ratio = fminf(target_ratio, expf(0.1f + 4.f * rsqrtf((float)k) + 3.f * slack));
  const float next = t_k * expf(-logf(ratio) / (alpha > 0.f ? alpha : 8.0f));
  st->tau = next > 0.f ? next : 0.f;
  st->aimed = (unsigned int)(ratio * (float)k);
  st->alpha = alpha;
  st->slack = slack;
  st->n_sel = n_sel;
  st->n_cand = count;
  st->fallback = exact ? 1u : 0u;
  if (exact) st->n_fallbacks = was.n_fallbacks + 1u;
  st->kth_mag = t_k;
  st->n_calls = was.stream_calls;
}

// Ranks the entries put aside, one per thread: the first k_rem go to the list from pos0 on, the others back to r.
// Returns the k_rem-th key.  One CTA; the list is complete.
__device__ __forceinline__ uint32_t settle_aside(PickShared& s, float* r, const Winners& out, unsigned int pos0,
                                                 unsigned int k_rem) {
  const unsigned int n = s.aside_n, t = threadIdx.x;
  if (t < n) {
    const uint32_t key = s.aside_key[t];
    unsigned int rank = 0;
    for (unsigned int u = 0; u < n; u += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(&s.aside_key[u]);
      rank += (u < n && (q.x > key || (q.x == key && u < t))) ? 1u : 0u;
      rank += (u + 1 < n && (q.y > key || (q.y == key && u + 1 < t))) ? 1u : 0u;
      rank += (u + 2 < n && (q.z > key || (q.z == key && u + 2 < t))) ? 1u : 0u;
      rank += (u + 3 < n && (q.w > key || (q.w == key && u + 3 < t))) ? 1u : 0u;
    }
    const Pair e = s.aside[t];
    if (rank < k_rem) out.put(pos0 + rank, e);
    else r[e.idx] = e.val;
    if (rank + 1u == k_rem) s.kth = key;
  }
  __syncthreads();
  return s.kth;
}

constexpr int kSmallRegs = kPickSmall / kPickThreads;  // candidates per thread in registers: one CTA
constexpr int kSweep = 8;  // candidates per thread and round of the sweep over all CTAs
// Least share of a CTA in that sweep.  (1 024, 2 048 and 4 096: compress of 8 M at 0.005 34.4, 35.2 and 37.1 us, select
// of 16 M at 0.001 45.8, 46.1 and 47.0; without a bound 8 M at 0.002 is 1 us slower.)
constexpr unsigned int kMinShare = 1024u;
constexpr int kClusterRegs = kPickCluster / (kPickCtas * kPickThreads);  // and the cluster
constexpr unsigned int kPickChunk = 4u * kPickThreads; // candidates per ticket, where they are counted or put back
constexpr int kExactVec = 4;                           // float4 of r per thread and ticket in exact mode
constexpr unsigned int kExactChunk = kExactVec * 4u * kPickThreads;

// k <= C <= kPickSmall: one CTA, candidates in registers, nothing but the list itself in global memory.
// Latency-bound (about 1 000 to 4 000 entries): what counts is the number of dependent steps.
__device__ __forceinline__ uint32_t pick_small(PickShared& s, float* r, const Pair* cand, const Winners& out,
                                               unsigned int k, unsigned int C, Level lv, Pair ahead) {
  Pair c[kSmallRegs];
  c[0] = ahead;
#pragma unroll
  for (int j = 1; j < kSmallRegs; ++j) {
    const unsigned int i = (unsigned int)j * kPickThreads + threadIdx.x;
    c[j].idx = 0;
    c[j].val = 0.f;
    if (i < C) c[j] = ld_pair_cg(&cand[i]);
  }
  auto live = [&](int j) { return (unsigned int)j * kPickThreads + threadIdx.x < C; };
  unsigned int k_rem = k;
  bool aside = false;  // the entries of the threshold's bin (5 to 50 after one level) are ranked directly
  for (;;) {
    *my_bins(s) = make_uint2(0u, 0u);
    if (threadIdx.x == 0) s.tie = s.aside_n = 0u;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSmallRegs; ++j)
      if (live(j) && lv.has(mag_key(c[j].val))) atomicAdd(&s.hist[lv.bin(mag_key(c[j].val))], 1u);
    __syncthreads();
    find_bin(s, *my_bins(s), k_rem);
    k_rem = s.res_krem;
    if (!lv.narrow(s.res_bin)) break;
    if (s.res_n <= kAside) {
      aside = true;
      break;
    }
  }
  const uint32_t th = lv.lo, top = lv.hi;
  unsigned int won = 0, gone = 0, n = 0;
#pragma unroll
  for (int j = 0; j < kSmallRegs; ++j) {
    if ((unsigned int)j * kPickThreads >= C) break;
    const uint32_t key = mag_key(c[j].val);
    bool win;
    if (aside) {
      win = live(j) && key > top;
      if (live(j) && key >= th && !win) {
        const unsigned int at = atomicAdd(&s.aside_n, 1u);
        s.aside_key[at] = key;
        s.aside[at] = c[j];
        gone |= 1u << j;
      }
    } else {
      win = passes(live(j), key, th, k_rem, &s.tie);
    }
    if (win) {
      won |= 1u << j;
      ++n;
    }
  }
  unsigned int pos = place(s, n, nullptr, 0u);
#pragma unroll
  for (int j = 0; j < kSmallRegs; ++j) {
    if (!live(j)) break;
    if (won & (1u << j)) out.put(pos++, c[j]);
    else if (!(gone & (1u << j))) r[c[j].idx] = c[j].val;
  }
  return aside ? settle_aside(s, r, out, k - k_rem, k_rem) : th;
}

// kPickSmall < C <= kPickCluster: the same with 8 CTAs that meet in the hardware barrier (0.2 us) and add
// up their counts over distributed shared memory.  Every CTA of the first cluster calls this.
__device__ __forceinline__ uint32_t pick_cluster(PickShared& s, float* r, const Pair* cand, const Winners& out,
                                                 unsigned int k, unsigned int C, Level lv) {
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const unsigned int rank = cluster.block_rank();
  constexpr unsigned int kStride = (unsigned int)kPickCtas * kPickThreads;
  static_assert(kClusterRegs * kStride == kPickCluster, "every candidate has a register");
  const unsigned int lane0 = rank * kPickThreads + threadIdx.x;
  const unsigned int trips = (C + kStride - 1u) / kStride;
  Pair c[kClusterRegs];
#pragma unroll
  for (int j = 0; j < kClusterRegs; ++j) {
    const unsigned int i = (unsigned int)j * kStride + lane0;
    c[j].idx = -1;
    c[j].val = 0.f;
    if (i < C) c[j] = ld_pair_cg(&cand[i]);
  }
  unsigned int k_rem = k;
  bool aside = false;  // as with one CTA; the list is in CTA 0, complete with the barrier that tells the totals
  int buf = 0;
  for (;;) {
    *my_bins(s) = make_uint2(0u, 0u);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kClusterRegs; ++j) {
      if ((unsigned int)j >= trips) break;
      const uint32_t key = mag_key(c[j].val);
      if (c[j].idx >= 0 && lv.has(key)) atomicAdd(&s.hist[lv.bin(key)], 1u);
    }
    __syncthreads();
    // Bin b is summed up in CTA b mod 8.  (Reading all eight histograms in every CTA moves 64 KB per SM over
    // the cluster network: 2 us per level.)  The next level's buffer is cleared here: it was read two levels
    // ago, before the barrier that this CTA has passed since, and is added to after the barrier below.
    const uint2 part = *my_bins(s);
    const unsigned int b0 = 2u * threadIdx.x;
    if (part.x) atomicAdd(cluster.map_shared_rank(&s.share[buf][b0 / kPickCtas], b0 % kPickCtas), part.x);
    if (part.y) atomicAdd(cluster.map_shared_rank(&s.share[buf][b0 / kPickCtas], b0 % kPickCtas + 1u), part.y);
    const int next = buf == 2 ? 0 : buf + 1;
    if (threadIdx.x < (unsigned int)(kBins / kPickCtas)) s.share[next][threadIdx.x] = 0u;
    cluster_barrier();
    uint2 sum;
    sum.x = *cluster.map_shared_rank(&s.share[buf][b0 / kPickCtas], b0 % kPickCtas);
    sum.y = *cluster.map_shared_rank(&s.share[buf][b0 / kPickCtas], b0 % kPickCtas + 1u);
    find_bin(s, sum, k_rem);
    k_rem = s.res_krem;
    if (!lv.narrow(s.res_bin)) break;
    if (s.res_n <= kAside) {
      aside = true;
      break;
    }
    buf = next;
  }
  const uint32_t th = lv.lo, top = lv.hi;
  unsigned int* const tie = cluster.map_shared_rank(&s.tie, 0);
  unsigned int won = 0, n = 0;
#pragma unroll
  for (int j = 0; j < kClusterRegs; ++j) {
    if ((unsigned int)j >= trips) break;
    const uint32_t key = mag_key(c[j].val);
    bool win;
    if (aside) {
      win = c[j].idx >= 0 && key > top;
      if (c[j].idx >= 0 && key >= th && !win) {
        const unsigned int at = atomicAdd(cluster.map_shared_rank(&s.aside_n, 0), 1u);
        *cluster.map_shared_rank(&s.aside_key[at], 0) = key;
        *cluster.map_shared_rank(&s.aside[at], 0) = c[j];
        c[j].idx = -1;
      }
    } else {
      win = passes(c[j].idx >= 0, key, th, k_rem, tie);
    }
    if (win) {
      won |= 1u << j;
      ++n;
    }
  }
  unsigned int pos = place(s, n, nullptr, 0u);
  // the CTA's total to everybody (nobody reads another CTA's memory after this barrier, so CTAs may leave)
  if (threadIdx.x == kPickThreads - 1) s.base[0] = pos + n;
  __syncthreads();
  if (threadIdx.x < (unsigned int)kPickCtas) *cluster.map_shared_rank(&s.cta_n[rank], threadIdx.x) = s.base[0];
  cluster_barrier();
  for (unsigned int q = 0; q < rank; ++q) pos += s.cta_n[q];
#pragma unroll
  for (int j = 0; j < kClusterRegs; ++j) {
    if (c[j].idx < 0) continue;
    if (won & (1u << j)) out.put(pos++, c[j]);
    else r[c[j].idx] = c[j].val;
  }
  return aside && rank == 0u ? settle_aside(s, r, out, k - k_rem, k_rem) : th;
}

// counted: the first level of the candidates has been counted by the stream pass.  WIDE: launched without clusters,
// otherwise in clusters of kPickCtas.
template <bool WIDE>
__device__ __forceinline__ void pick(PickShared& s, float* r, long long d, const Pair* cand, unsigned int cap,
                                     const Winners& out, unsigned int k, K1State* st, Ctrl* ctrl_pair, int counted,
                                     float target_ratio, unsigned long long limit_ns) {
  // what the cluster's CTAs add to in one another, ready before the stream pass has ended
  if (threadIdx.x == 0) s.tie = s.aside_n = 0u;
  if (!WIDE) {
    if (threadIdx.x < (unsigned int)(kBins / kPickCtas)) s.share[0][threadIdx.x] = 0u;
    cluster_barrier();
  }
  pdl_begin(r, cand, st, ctrl_pair);
  // one round of loads: the call's parity, both blocks' counts, and (unseen) the first candidates
  K1State was;
  was.stream_calls = st->stream_calls;
  was.tau = st->tau;
  was.kth_mag = st->kth_mag;
  was.alpha = st->alpha;
  was.slack = st->slack;
  was.aimed = st->aimed;
  was.n_fallbacks = st->n_fallbacks;
  const unsigned int calls = was.stream_calls - 1u;
  const unsigned int n_out[2] = {__ldcg(&ctrl_pair[0].n_out), __ldcg(&ctrl_pair[1].n_out)};
  uint2 level[2];  // WIDE (and so counted): the first level of either block
  if (WIDE) {
    level[0] = global_counts(ctrl_pair[0].hist[0][0]);
    level[1] = global_counts(ctrl_pair[1].hist[0][0]);
  }
  Pair ahead;
  ahead.idx = 0;
  ahead.val = 0.f;
  if (!WIDE && blockIdx.x == 0 && threadIdx.x < cap) ahead = ld_pair_cg(&cand[threadIdx.x]);
  Ctrl* const ctrl = ctrl_pair + (calls & 1u);
  const unsigned int count = n_out[calls & 1u];
  const unsigned int C = count < cap ? count : cap;
  const bool exact_mode = (count > cap) || (C < k);
  trace_stamp(ctrl, 2);
  const Bands bands = first_bands(was.tau, was.kth_mag);
  Level lv{bands.lo, 0x7fffffffu, bands.shift, true};
  uint32_t th = 0u;

  if (!WIDE && !exact_mode && C <= kPickCluster) {
    if (C <= kPickSmall) {
      if (blockIdx.x != 0) return;
      th = pick_small(s, r, cand, out, k, C, lv, ahead);
    } else {
      if (blockIdx.x >= (unsigned int)kPickCtas) return;
      th = pick_cluster(s, r, cand, out, k, C, lv);
      if (blockIdx.x != 0) return;
    }
    trace_stamp(ctrl, 4);
    if (threadIdx.x == 0) finish_state(st, was, th, k, k, count, C, false, target_ratio);
    return;
  }

  int ph = 0;
  unsigned int k_rem = k;
  if (!exact_mode) {
    // The candidates shared out over all CTAs.  The first level was counted by the stream pass (counted) or is counted
    // here, in chunks.  As a rule the threshold's bin then holds few enough entries (300 to 1 400) to leave them to
    // one CTA: a single sweep sends what lies above the bin to the list, returns what lies below to r, and puts what
    // lies in it aside; the CTA that finishes the sweep picks among those (against a level and a sweep more: whole
    // call at 25.6 M and 0.01 63.9 -> 60.6 us, 66 M and 0.01 148.6 -> 144.2, 138 M and 0.01 294 -> 288).
    // A bin with more is counted by finer levels, a phase each.
    const unsigned int share = max((C + gridDim.x - 1u) / gridDim.x, kMinShare), nshares = (C + share - 1u) / share;
    const unsigned int begin = blockIdx.x * share, end = begin + share < C ? begin + share : C;
    if (begin >= end) return;  // (from here on the call does not end without this CTA, however late it has started)
    const unsigned int nchunks = (C + kPickChunk - 1u) / kPickChunk;
    unsigned int* level_hist = ctrl->hist[0][0];
    bool have = counted != 0, aside = false;
    int row = 0;
    for (;;) {
      if (!have) {
        *my_bins(s) = make_uint2(0u, 0u);
        const unsigned int mine = for_chunks(s, ctrl, ph, nchunks, [&](unsigned int chunk) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const unsigned int i = chunk * kPickChunk + (unsigned int)j * kPickThreads + threadIdx.x;
            if (i >= C) break;
            const uint32_t key = mag_key(ld_pair_cg(&cand[i]).val);
            if (lv.has(key)) atomicAdd(&s.hist[lv.bin(key)], 1u);
          }
        });
        if (mine) publish_hist(s, level_hist);
        report(ctrl, ph, mine, nchunks);
        if (!wait_phase(s, ctrl, ph, nchunks, limit_ns, 100 + ph)) return;  // (every CTA has a share of the sweep)
        ++ph;
      }
      have = false;
      uint2 counts;
      if (WIDE && ph == 0) counts = (calls & 1u) ? level[1] : level[0];
      else counts = global_counts(level_hist);
      find_bin(s, counts, k_rem);
      k_rem = s.res_krem;
      if (!lv.narrow(s.res_bin)) break;
      if (s.res_n <= kPickSmall) {
        aside = true;
        break;
      }
      level_hist = ctrl->hist[0][++row];
      __syncthreads();
    }
    th = lv.lo;
    const uint32_t top = aside ? lv.hi : lv.lo;
    Pair* const between = reinterpret_cast<Pair*>(ctrl->hist[2]);  // (rows that K1 has no other use for)
    static_assert(sizeof(ctrl->hist[2]) >= kPickSmall * sizeof(Pair), "room for the entries put aside");
    if (threadIdx.x == 0) ctrl->trace[3] = globaltimer_ns();  // k-th magnitude known, or its bin
    // The sweep.  Every CTA has an equal share, up to kSweep entries per thread in flight, and one place in the list
    // for all of a round's winners.  Nobody waits for anybody here, so the shares need no tickets.  (Chunks of 4 096
    // by tickets were 9 us each, a chain of a ticket, a load, a place and the barriers between them; and in clusters,
    // as the kernel was launched for every size, 112 of its 152 CTAs ran side by side.  select + update of 60 M at
    // 0.007 153.2 -> 149.2 us, 16 M at 0.005 51.0 -> 49.7, 5 M at 0.01 26.8 -> 25.9; compress, which writes three
    // lists, 4 M at 0.008 27.1 -> 22.9, 8 M at 0.005 38.5 -> 34.5, 30 M at 0.002 93.3 -> 88.6.)
    unsigned int turn = 0;
    for (unsigned int base = begin; base < end; base += (unsigned int)kSweep * kPickThreads) {
      Pair c[kSweep];
      unsigned int won = 0, n = 0;
#pragma unroll
      for (int j = 0; j < kSweep; ++j) {
        const unsigned int i = base + (unsigned int)j * kPickThreads + threadIdx.x;
        c[j].idx = -1;
        c[j].val = 0.f;
        if (i < end) c[j] = ld_pair_cg(&cand[i]);
      }
#pragma unroll
      for (int j = 0; j < kSweep; ++j) {
        const uint32_t key = mag_key(c[j].val);
        bool win;
        if (aside) {
          win = c[j].idx >= 0 && key > top;
          if (c[j].idx >= 0 && key >= th && !win) {
            const unsigned int at = atomicAdd(&ctrl->live[0], 1u);
            if (at < kPickSmall) st_pair(&between[at], c[j]);
            c[j].idx = -1;
          }
        } else {
          win = passes(c[j].idx >= 0, key, th, k_rem, &ctrl->tie[0]);
        }
        if (win) won |= 1u << j;
        n += (unsigned int)__popc(__ballot_sync(0xffffffffu, win));
      }
      unsigned int pos = place_warp(s, n, &ctrl->cursor[0], turn++);
#pragma unroll
      for (int j = 0; j < kSweep; ++j) {
        const bool win = (won & (1u << j)) != 0u;
        const unsigned int m = __ballot_sync(0xffffffffu, win);
        if (win) {
          const unsigned int at = pos + __popc(m & lanemask_lt());
          if (at < k) out.put(at, c[j]);
        } else if (c[j].idx >= 0) {
          r[c[j].idx] = c[j].val;
        }
        pos += (unsigned int)__popc(m);
      }
    }
    const bool last = report(ctrl, ph, 1u, nshares);
    if (aside) {
      if (threadIdx.x == 0) s.ok = last ? 1 : 0;
      __syncthreads();
      if (!s.ok) return;
      __threadfence();
      const unsigned int n = __ldcg(&ctrl->live[0]);
      Pair front;
      front.idx = 0;
      front.val = 0.f;
      if (threadIdx.x < n) front = ld_pair_cg(&between[threadIdx.x]);
      th = pick_small(s, r, between, out.from(k - k_rem), k_rem, n, lv, front);
    }
    if (last) {
      finish_state(st, was, th, k, k, count, C, false, target_ratio);
      ctrl->trace[4] = globaltimer_ns();  // all winners compacted
    }
    return;
  }

  // ---- exact mode
  if (C) {  // the stream pass took these out of the residual
    const unsigned int nchunks = (C + kPickChunk - 1u) / kPickChunk;
    const unsigned int mine = for_chunks(s, ctrl, ph, nchunks, [&](unsigned int chunk) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned int i = chunk * kPickChunk + (unsigned int)j * kPickThreads + threadIdx.x;
        if (i >= C) break;
        const Pair e = ld_pair_cg(&cand[i]);
        r[e.idx] = e.val;
      }
    });
    report(ctrl, ph, mine, nchunks);  // (a CTA without a chunk of this short phase stays for the sweeps)
    if (!wait_phase(s, ctrl, ph, nchunks, limit_ns, 110)) return;
    ++ph;
  }
  const unsigned int mis = (unsigned int)((reinterpret_cast<uintptr_t>(r) >> 2) & 3u);
  long long head = mis ? (4 - mis) : 0;
  if (head > d) head = d;
  const unsigned int nvec = (unsigned int)((d - head) >> 2);
  const float4* r4 = reinterpret_cast<const float4*>(r + head);
  const unsigned int nscalar = (unsigned int)(d - ((long long)nvec << 2));   // head and tail, at most 6
  const unsigned int nchunks = (unsigned int)((d + kExactChunk - 1) / kExactChunk);
  // this thread's float4 u of a chunk (out of range: ok = false), and chunk 0's scalar
  auto vec_at = [&](unsigned int chunk, int u) { return chunk * (kExactChunk / 4u) + (unsigned int)u * kPickThreads + threadIdx.x; };
  auto scalar_at = [&](unsigned int chunk) -> long long {
    if (chunk != 0u || threadIdx.x >= nscalar) return -1;
    const long long j = threadIdx.x;
    return j < head ? j : head + ((long long)nvec << 2) + (j - head);
  };
  unsigned int quota = 0xffffffffu;  // d <= k: everything is selected
  if (d > (long long)k) {
    lv = Level{0u, 0x7fffffffu, 20u, false};
    int row = 0;
    for (;;) {
      *my_bins(s) = make_uint2(0u, 0u);
      const unsigned int mine = for_chunks(s, ctrl, ph, nchunks, [&](unsigned int chunk) {
        float4 x[kExactVec];
#pragma unroll
        for (int u = 0; u < kExactVec; ++u) {
          const unsigned int v = vec_at(chunk, u);
          if (v < nvec) x[u] = __ldcg(&r4[v]);
        }
        auto count_key = [&](float a) {
          if (lv.has(mag_key(a))) atomicAdd(&s.hist[lv.bin(mag_key(a))], 1u);
        };
#pragma unroll
        for (int u = 0; u < kExactVec; ++u) {
          if (vec_at(chunk, u) >= nvec) break;
          count_key(x[u].x);
          count_key(x[u].y);
          count_key(x[u].z);
          count_key(x[u].w);
        }
        const long long i = scalar_at(chunk);
        if (i >= 0) count_key(__ldcg(&r[i]));
      });
      if (mine == 0u) return;  // those that hold chunks finish the call
      publish_hist(s, ctrl->hist[1][row]);
      report(ctrl, ph, mine, nchunks);
      if (!wait_phase(s, ctrl, ph, nchunks, limit_ns, 120 + ph)) return;
      ++ph;
      find_bin(s, global_counts(ctrl->hist[1][row]), k_rem);
      k_rem = s.res_krem;
      if (!lv.narrow(s.res_bin)) break;
      ++row;
      __syncthreads();
    }
    th = lv.lo;
    quota = k_rem;
  }
  unsigned int turn = 0;
  const unsigned int mine = for_chunks(s, ctrl, ph, nchunks, [&](unsigned int chunk) {
    float x[4 * kExactVec + 1];
    unsigned int won = 0, n = 0;
#pragma unroll
    for (int u = 0; u < kExactVec; ++u) {
      const unsigned int v = vec_at(chunk, u);
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
      if (v < nvec) y = __ldcg(&r4[v]);
      x[4 * u] = y.x;
      x[4 * u + 1] = y.y;
      x[4 * u + 2] = y.z;
      x[4 * u + 3] = y.w;
    }
    const long long is = scalar_at(chunk);
    x[4 * kExactVec] = is >= 0 ? __ldcg(&r[is]) : 0.f;
#pragma unroll
    for (int e = 0; e <= 4 * kExactVec; ++e) {
      const bool live = e < 4 * kExactVec ? vec_at(chunk, e >> 2) < nvec : is >= 0;
      if (passes(live, mag_key(x[e]), th, quota, &ctrl->tie[1])) {
        won |= 1u << e;
        ++n;
      }
    }
    unsigned int pos = place(s, n, &ctrl->cursor[1], turn++);
    if (n == 0u) return;
#pragma unroll
    for (int e = 0; e <= 4 * kExactVec; ++e) {
      if (!(won & (1u << e))) continue;
      const long long i = e < 4 * kExactVec ? head + 4ll * vec_at(chunk, e >> 2) + (e & 3) : is;
      Pair p;
      p.idx = (int32_t)i;
      p.val = x[e];
      if (pos < k) out.put(pos, p);
      ++pos;
      r[i] = 0.f;
    }
  });
  if (report(ctrl, ph, mine, nchunks)) {
    const unsigned int n_sel = d < (long long)k ? (unsigned int)d : k;
    finish_state(st, was, th, n_sel, k, count, C, true, target_ratio);
    ctrl->trace[5] = globaltimer_ns();
  }
}

__global__ void __cluster_dims__(kPickCtas, 1, 1) __launch_bounds__(kPickThreads, 1)
k1_pick(float* r, long long d, const Pair* cand, unsigned int cap, Winners out, unsigned int k, K1State* st,
        Ctrl* ctrl_pair, int counted, float target_ratio, unsigned long long limit_ns) {
  __shared__ __align__(16) PickShared s;
  pick<false>(s, r, d, cand, cap, out, k, st, ctrl_pair, counted, target_ratio, limit_ns);
}
__global__ void __launch_bounds__(kPickThreads, 1)
k1_pick_wide(float* r, long long d, const Pair* cand, unsigned int cap, Winners out, unsigned int k, K1State* st,
             Ctrl* ctrl_pair, int counted, float target_ratio, unsigned long long limit_ns) {
  __shared__ __align__(16) PickShared s;
  pick<true>(s, r, d, cand, cap, out, k, st, ctrl_pair, counted, target_ratio, limit_ns);
}

}  // namespace gtk

using namespace gtk;

extern "C" unsigned long long gtk_ctrl_bytes(void) { return sizeof(Ctrl); }

// Whether a select (compress: gtk_k1_compress) of k out of d elements launches its pick without clusters.  The candidates
// are 1.2 to 3 times k, and at most d.  One cluster picks from up to 32 K of them without a sweep over lists in memory;
// without clusters more CTAs share that sweep.  So clusters for every vector most of which fits one, and up to the k where
// the candidates of a short vector outgrow it; the longer the stream pass, the less the start of more CTAs shows behind
// it, and where each winner goes to three places 8 SMs are soon too few.  In clusters and without, us:
//   select + update   1.6 M at 0.01 16.1, 16.7   2 M at 0.01 18.0, 17.6   8 M at 0.002 31.2, 30.7
//                     13 M at 0.001 40.4, 40.0   25 M at 0.001 63.1, 62.2
//   select            25 K, k 18 001 12.9, 14.4   40 K, 27 000 14.1, 14.7; 36 000 14.8, 14.0
//                     60 K, 16 000 13.1, 14.0; 24 000 14.6, 14.2   100 K, 18 001 12.85, 13.6; 24 000 15.15, 14.3
//                     400 K, 18 001 13.3, 13.6; 24 000 14.0, 13.9   1 M, 13 000 13.7, 14.2; 18 001 14.55, 14.2
//                     2.9 M, 13 000 16.1, 16.2; 16 000 16.95, 16.6
//   compress          25 K, k 13 000 17.6, 18.5   60 K, 13 000 16.8, 18.0; 18 000 19.4, 18.6
//                     100 K, 15 000 17.4, 17.7; 18 000 18.5, 17.8   200 K, 15 000 18.1, 17.7   1 M, 13 000 22.7, 21.1
//                     8 M at 0.001 32.5, 34.1; at 0.002 36.0, 34.4   16 M at 0.0015 58.7, 55.1
extern "C" int gtk_k1_pick_is_wide(long long d, unsigned int k, int compress) {
  if (d < 3ll * kPickCluster / 2) return k > kPickCluster;
  if (compress) return k > (d < 200 * 1000 ? 16000u : kCountFrom);
  return k > (d < 800 * 1000 ? 22000u : d < 3 * 1000 * 1000 ? 18000u : kCountFrom);
}

namespace {
// Launches the two kernels; `stream_pass(counted, dynamic, grid)` launches the first.
template <typename Stream>
int k1_launch_with(Stream stream_pass, float* r, long long d, unsigned int k, Pair* cand, unsigned int cap, Winners out,
                   K1State* st, Ctrl* ctrl_pair, float target_ratio, unsigned long long limit_ns, cudaStream_t stream) {
  const DeviceInfo* di = gtk_device_info();
  if (!di) return GTK_ERR_CUDA;
  // Two float4 of each array per thread and tile in the static split (four: 2 % slower, a coarser last round),
  // four in the dynamic one (two: 2 % slower at 138 M).
  const long long full = 2ll * di->sms;
  const long long nvec = d / 4;
  const bool dynamic = nvec >= kDynamicMinVec;
  const long long tile = (long long)kK1Threads * (dynamic ? 4 : 2);
  long long grid = (nvec + tile - 1) / tile;
  grid = grid < 1 ? 1 : (grid > full ? full : grid);
  // The first level is counted on the fly where the candidates (1.2 to 3 times k) may be more than one cluster takes: it
  // saves their sweep a phase of counting by tickets, 2 us; below, the CTAs that pick count faster than the stream
  // pass publishes.
  const bool counted = k > kCountFrom;
  cudaError_t e = stream_pass(counted, dynamic, (int)grid);
  if (e != cudaSuccess) return GTK_ERR_CUDA;
  // The pick: as many CTAs as exact mode can use, or the sweep over many candidates.  Clusters only where a cluster may
  // pick: 8 CTAs that each fill an SM find a place only inside one GPC, and not on every SM of it.  Without them fewer
  // CTAs than SMs as long as the sweep is short, so that the call does not wait for CTAs on the SMs that end the stream
  // pass last (with 96, 118 and 148 of 148: select + update of 5 M at 0.01 25.2, 25.9 and 26.7 us, 16 M at 0.005 49.0,
  // 49.7 and 50.0), and as many as make exact mode no slower than in clusters (8 M at 0.002, a first call: 68.9, 61.8
  // and 57.7 us, in clusters 62.1; 30 M at 0.003 231, 203, 190 and 211).
  const bool wide = gtk_k1_pick_is_wide(d, k, out.dense != nullptr) != 0;
  long long ctas = (d + kExactChunk - 1) / kExactChunk;
  if (wide) {
    const long long most = di->sms * 4 / 5 + k / 8192;
    if (ctas < (long long)k / kPickThreads) ctas = (long long)k / kPickThreads;
    if (ctas > most) ctas = most;
  }
  if (ctas > di->sms) ctas = di->sms;
  if (!wide) ctas = (ctas + kPickCtas - 1) / kPickCtas * kPickCtas;
  e = launch_pdl(wide ? k1_pick_wide : k1_pick, (int)ctas, kPickThreads, stream, r, d, cand, cap, out, k, st, ctrl_pair,
                 counted ? 1 : 0, target_ratio, limit_ns);
  gtk_count_launch(2);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}

// out.dense: g itself (then it is left sparsified) or nullptr (then g is only read).
int k1_launch(const float* g_in, float* r, const float* g_scale, long long d, unsigned int k,
              Pair* cand, unsigned int cap, Winners out, K1State* st, Ctrl* ctrl_pair,
              float target_ratio, unsigned long long limit_ns, cudaStream_t stream) {
  float* g = const_cast<float*>(g_in);
  auto stream_pass = [&](bool counted, bool dynamic, int grid) {
    auto go = [&](auto zero) {
      constexpr bool Z = decltype(zero)::value;
      auto fn = dynamic ? (counted ? k1_stream<true, true, Z> : k1_stream<false, true, Z>)
                        : (counted ? k1_stream<true, false, Z> : k1_stream<false, false, Z>);
      return launch_pdl(fn, grid, kK1Threads, stream, g, r, g_scale, d, cand, cap, st, ctrl_pair);
    };
    return out.dense ? go(std::true_type{}) : go(std::false_type{});
  };
  return k1_launch_with(stream_pass, r, d, k, cand, cap, out, st, ctrl_pair, target_ratio, limit_ns, stream);
}

template <int N>
int k1_launch_segments(const unsigned long long* grads, unsigned int n, const unsigned int* segments, float* r, long long d,
                       unsigned int k, Pair* cand, unsigned int cap, Pair* sel, K1State* st, Ctrl* ctrl_pair,
                       float target_ratio, unsigned long long limit_ns, cudaStream_t stream) {
  GradPointers<N> g;
  for (unsigned int i = 0; i < n; ++i) g.g[i] = reinterpret_cast<const float*>(static_cast<uintptr_t>(grads[i]));
  auto stream_pass = [&](bool counted, bool dynamic, int grid) {
    auto fn = dynamic ? (counted ? k1_stream_segments<true, true, N> : k1_stream_segments<false, true, N>)
                      : (counted ? k1_stream_segments<true, false, N> : k1_stream_segments<false, false, N>);
    return launch_pdl(fn, grid, kK1Threads, stream, g, segments, n, r, d, cand, cap, st, ctrl_pair);
  };
  return k1_launch_with(stream_pass, r, d, k, cand, cap, Winners{sel, nullptr, nullptr, nullptr}, st, ctrl_pair, target_ratio,
                        limit_ns, stream);
}
}  // namespace

static bool k1_args_ok(const float* g, const float* r, long long d, unsigned int k, unsigned int cap) {
  if (d <= 0 || d >= (1ll << 31) || k == 0 || k > cap) return false;
  // g and r must share their offset inside a 16-byte line (same flat layout)
  return (reinterpret_cast<uintptr_t>(g) & 15u) == (reinterpret_cast<uintptr_t>(r) & 15u) &&
         (reinterpret_cast<uintptr_t>(r) & 3u) == 0u;
}

// ctrl: TWO consecutive control blocks (2 * gtk_ctrl_bytes()), zero when first used.
extern "C" int gtk_k1_select(const float* g, float* r, const float* g_scale, long long d,
                             unsigned int k, void* cand, unsigned int cap, void* sel, void* state,
                             void* ctrl, float target_ratio, unsigned long long limit_ns,
                             void* stream_) {
  if (!k1_args_ok(g, r, d, k, cap)) return GTK_ERR_ARG;
  return k1_launch(g, r, g_scale, d, k, (Pair*)cand, cap, Winners{(Pair*)sel, nullptr, nullptr, nullptr}, (K1State*)state,
                   (Ctrl*)ctrl, target_ratio, limit_ns, (cudaStream_t)stream_);
}

// The select with the gradient in n tensors instead of one vector: grads[s] (device address, 0: no gradient) belongs
// to the elements that segments (device memory: n + 1 start positions in float4, ascending from 0, the last one
// ceil(d / 4); n lengths in elements) gives segment s.  r must be 16-byte aligned, n at most 1024.
extern "C" int gtk_k1_select_segments(gtk_addresses grads, const unsigned int* segments, float* r, long long d,
                                      unsigned int k, void* cand, unsigned int cap, void* sel, void* state, void* ctrl,
                                      float target_ratio, unsigned long long limit_ns, void* stream_) {
  if (!k1_args_ok(r, r, d, k, cap) || (reinterpret_cast<uintptr_t>(r) & 15u) || grads.n == 0) return GTK_ERR_ARG;
  auto go = [&](auto n) {
    return k1_launch_segments<decltype(n)::value>(grads.p, grads.n, segments, r, d, k, (Pair*)cand, cap, (Pair*)sel,
                                                  (K1State*)state, (Ctrl*)ctrl, target_ratio, limit_ns,
                                                  (cudaStream_t)stream_);
  };
  // (the pointers are kernel parameters, so that a captured launch carries them)
  if (grads.n <= 64) return go(std::integral_constant<int, 64>{});
  if (grads.n <= 256) return go(std::integral_constant<int, 256>{});
  if (grads.n <= 1024) return go(std::integral_constant<int, 1024>{});
  return GTK_ERR_ARG;
}

// The select, with g left sparsified (selected entries keep g + r, all others are 0) and the selection also
// as int64 indices and fp32 values, min(k, d) of each.
extern "C" int gtk_k1_compress(float* g, float* r, long long d, unsigned int k, void* cand, unsigned int cap, void* sel,
                               void* state, void* ctrl, float target_ratio, unsigned long long limit_ns,
                               long long* idx_out, float* val_out, void* stream_) {
  if (!k1_args_ok(g, r, d, k, cap) || !idx_out || !val_out) return GTK_ERR_ARG;
  return k1_launch(g, r, nullptr, d, k, (Pair*)cand, cap, Winners{(Pair*)sel, g, idx_out, val_out}, (K1State*)state,
                   (Ctrl*)ctrl, target_ratio, limit_ns, (cudaStream_t)stream_);
}

// ---------------------------------------------------------------------------
// Allocation-free variant (declared and documented in k1_select_noalloc.h).
// The scratch that gtk_k1_select takes from its caller lives here in a static
// device array; the kernels are the ones above, unchanged.
// ---------------------------------------------------------------------------
#include <mutex>
#include "k1_select_noalloc.h"

namespace {

constexpr unsigned int kNoAllocMaxK = 16384u;
constexpr unsigned int kNoAllocCap = 131072u;                         // candidate pairs (8 x max k)
constexpr size_t kNoAllocCtrlOff = 0;                                  // two control blocks
constexpr size_t kNoAllocStateOff = (2 * sizeof(Ctrl) + 255) / 256 * 256;
constexpr size_t kNoAllocCandOff = kNoAllocStateOff + 256;
constexpr size_t kNoAllocBytes = kNoAllocCandOff + (size_t)kNoAllocCap * sizeof(Pair);

// In host code this name is only a handle for cudaGetSymbolAddress, never an address.
// Static device storage starts zeroed, which is what the control blocks need on first use.
static __device__ __align__(256) unsigned char g_k1_noalloc_scratch[kNoAllocBytes];

// Forget the predicted threshold.  The call counter is left alone: it decides which
// control block is clean.
__global__ void k1_noalloc_reset_state(K1State* st) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    st->tau = __int_as_float(0x7f800000);  // +inf: the next call takes the exact path
    st->n_sel = 0u;
    st->n_cand = 0u;
    st->fallback = 0u;
    st->kth_mag = 0.f;
    st->aimed = 0u;
    st->alpha = 0.f;
  }
}

__global__ void k1_noalloc_publish_count(const K1State* st, unsigned int* n_sel_out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *n_sel_out = st->n_sel;
}

struct NoAllocDevice {
  unsigned char* base = nullptr;  // device address of g_k1_noalloc_scratch on this device
};
std::mutex g_noalloc_mu;
NoAllocDevice g_noalloc_dev[64];

}  // namespace

extern "C" unsigned int gtk_k1_noalloc_max_k(void) { return kNoAllocMaxK; }
extern "C" unsigned long long gtk_k1_noalloc_scratch_bytes(void) { return kNoAllocBytes; }

extern "C" int gtk_k1_select_noalloc(const float* g, float* r, long long d, unsigned int k,
                                     void* sel_out, unsigned int* n_sel_out, int reset_threshold,
                                     void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (k > kNoAllocMaxK) return GTK_ERR_TOO_LARGE;
  if (d <= 0 || d >= (1ll << 31) || k == 0 || !g || !r || !sel_out) return GTK_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(g) & 15u) != (reinterpret_cast<uintptr_t>(r) & 15u) ||
      (reinterpret_cast<uintptr_t>(r) & 3u) != 0u)
    return GTK_ERR_ARG;
  // pairs are stored with one 8-byte access, the count with a 4-byte one
  if ((reinterpret_cast<uintptr_t>(sel_out) & 7u) != 0u ||
      (n_sel_out && (reinterpret_cast<uintptr_t>(n_sel_out) & 3u) != 0u))
    return GTK_ERR_ARG;
  const DeviceInfo* di = gtk_device_info();
  if (!di || di->device < 0 || di->device >= 64) return GTK_ERR_CUDA;
  NoAllocDevice dev;
  bool first = false;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoAllocDevice& slot = g_noalloc_dev[di->device];
    if (!slot.base) {
      // once per device, with that device current
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_k1_noalloc_scratch) != cudaSuccess || !p) return GTK_ERR_CUDA;
      slot.base = static_cast<unsigned char*>(p);
      first = true;
    }
    dev = slot;
  }
  Ctrl* ctrl_pair = reinterpret_cast<Ctrl*>(dev.base + kNoAllocCtrlOff);
  K1State* st = reinterpret_cast<K1State*>(dev.base + kNoAllocStateOff);
  Pair* cand = reinterpret_cast<Pair*>(dev.base + kNoAllocCandOff);
  if (first || reset_threshold) {
    k1_noalloc_reset_state<<<1, 32, 0, stream>>>(st);
    gtk_count_launch(1);
  }
  // What must start at zero -- the control block of this call -- was cleared by the previous call
  // (or is still in its initial zero state); the candidate list is overwritten before it is read.
  const int code = k1_launch(g, r, nullptr, d, k, cand, kNoAllocCap,
                             Winners{static_cast<Pair*>(sel_out), nullptr, nullptr, nullptr}, st, ctrl_pair, 3.0f, 2000000000ull, stream);
  if (code != GTK_OK) return code;
  if (n_sel_out) {
    k1_noalloc_publish_count<<<1, 32, 0, stream>>>(st, n_sel_out);
    gtk_count_launch(1);
  }
  return cudaGetLastError() == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}

// Status of the shared scratch on the current device: out_status_where[0] = status code of the first
// failure recorded in either control block (0: none; the codes of gtk::Status), [1] = its code
// location.  With reset != 0 both control blocks and the threshold state are cleared afterwards, which
// is what brings the entry point back after a failed call (a barrier that ran into its limit leaves
// its control block marked aborted).  Copies 16 bytes to the host and waits for `stream` only; no
// allocation.  Returns GTK_ERR_ARG before the first gtk_k1_select_noalloc call on this device.
extern "C" int gtk_k1_noalloc_status(unsigned int* out_status_where, int reset, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  const DeviceInfo* di = gtk_device_info();
  if (!di || di->device < 0 || di->device >= 64) return GTK_ERR_CUDA;
  NoAllocDevice dev;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    dev = g_noalloc_dev[di->device];
  }
  if (!dev.base) return GTK_ERR_ARG;
  Ctrl* ctrl_pair = reinterpret_cast<Ctrl*>(dev.base + kNoAllocCtrlOff);
  unsigned int words[2][2] = {{0u, 0u}, {0u, 0u}};
  for (int b = 0; b < 2; ++b)
    if (cudaMemcpyAsync(words[b], &ctrl_pair[b].status, 2 * sizeof(unsigned int), cudaMemcpyDeviceToHost,
                        stream) != cudaSuccess)
      return GTK_ERR_CUDA;
  if (reset) {
    if (cudaMemsetAsync(ctrl_pair, 0, 2 * sizeof(Ctrl), stream) != cudaSuccess) return GTK_ERR_CUDA;
    k1_noalloc_reset_state<<<1, 32, 0, stream>>>(reinterpret_cast<K1State*>(dev.base + kNoAllocStateOff));
    gtk_count_launch(1);
  }
  if (cudaStreamSynchronize(stream) != cudaSuccess) return GTK_ERR_CUDA;
  const int b = words[0][0] ? 0 : 1;
  if (out_status_where) {
    out_status_where[0] = words[b][0];
    out_status_where[1] = words[b][1];
  }
  return GTK_OK;
}
