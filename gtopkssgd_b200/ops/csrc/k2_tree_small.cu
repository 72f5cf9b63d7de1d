// K2 for small sets: the gTop-k tree exchange with one CTA per rank, the current
// set in shared memory, and flags that travel with the data.
//
// Same semantics and failure rules as k2_gtopk_exchange.cu, for k up to kLLMaxK.
// A small exchange is a chain of short dependent steps, so this form takes out the
// long ones (per tree round at k = 1 000, before: 7 us of work and 2 to 3 us from
// sender to receiver):
//   * a sent entry is one 16-byte store {index, epoch, value, epoch}; the receiver's
//     thread polls exactly its entries.  No fence that waits for the stores to be
//     acknowledged, no flag behind them, no load after the flag.  Each 8-byte half
//     carries its own epoch, because only 8 bytes are written as one.
//   * the union lives in two dense arrays (this rank's entries, then the partner's) with an
//     open-addressing table of their indices, so an arriving entry meets its match in one
//     or two shared-memory probes instead of three trips to L2;
//   * the first selection level is counted while entries arrive, over a band above the
//     previous threshold; the few entries of the threshold's bin are ranked directly.
// (Keeping the entries in the table itself and marking the losers dead there was slower:
// every sweep then visits all slots, 8 per thread at k = 1 000, 5 us per selection.)
#include <atomic>
#include "exchange_common.cuh"
#include "launch.cuh"
#include "pick_common.cuh"

namespace gtk {

constexpr uint32_t kEmpty = 0xffffffffu;  // no index: d < 2^31
constexpr unsigned int kRankList = 32u;   // entries of the threshold's bin that are ranked directly

struct SmallShared : WideShared {
  unsigned int tie;
  unsigned int fresh_n;     // entries of the union that are not sums onto another
  unsigned int list_n;
  uint32_t list[kRankList];
  int ok;
};
// For a set size k: 2k entries (index, value), and at least twice as many table slots (index, position), three
// times where there is room: what counts is the longest probe sequence in a warp.
__host__ __device__ constexpr unsigned int small_slots(unsigned int k) {
  unsigned int n = 1024u;
  while (n < 6u * k) n *= 2u;
  return n;
}
constexpr size_t small_smem_bytes(unsigned int k) {
  return (sizeof(SmallShared) + 15) / 16 * 16 + 16ull * (k + 3) + 8ull * small_slots(k);
}

// Shared-memory accesses by 32-bit address.
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t shared_load(uint32_t a) {
  uint32_t v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void shared_store(uint32_t a, uint32_t v) {
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t shared_cas(uint32_t a, uint32_t was, uint32_t v) {
  uint32_t old;
  asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;" : "=r"(old) : "r"(a), "r"(was), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void shared_add(uint32_t a, uint32_t v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Index -> position in the dense arrays: two words per slot.
struct Table {
  uint32_t at;         // shared address of the slots
  unsigned int slots;  // a power of two
  int shift;           // 32 - log2(slots)

  // Multiplicative hashing with the golden ratio (Knuth, The Art of Computer Programming 3, 6.4).
  __device__ __forceinline__ unsigned int start(uint32_t idx) const { return (idx * 0x9e3779b1u) >> shift; }
  __device__ __forceinline__ unsigned int next(unsigned int s) const { return (s + 1u) & (slots - 1u); }
  // Enters idx at position `pos`, or returns the position it has.  (At half load the probing always ends.)
  // At most one thread enters a given index between two barriers.
  __device__ __forceinline__ unsigned int enter(uint32_t idx, unsigned int pos) const {
    for (unsigned int s = start(idx);; s = next(s)) {
      uint32_t w = shared_load(at + 4u * s);
      if (w == kEmpty) {
        w = shared_cas(at + 4u * s, kEmpty, idx);
        if (w == kEmpty) {
          shared_store(at + 4u * (slots + s), pos);
          return pos;
        }
      }
      if (w == idx) return shared_load(at + 4u * (slots + s));
    }
  }
  // The position of idx, kEmpty if it is not there.
  __device__ __forceinline__ unsigned int find(uint32_t idx) const {
    for (unsigned int s = start(idx);; s = next(s)) {
      const uint32_t w = shared_load(at + 4u * s);
      if (w == idx) return shared_load(at + 4u * (slots + s));
      if (w == kEmpty) return kEmpty;
    }
  }
};

__device__ __forceinline__ void ll_store(ulonglong2* p, Pair e, uint32_t epoch) {
  const unsigned long long tag = (unsigned long long)epoch << 32;
  asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(tag | (uint32_t)e.idx),
               "l"(tag | __float_as_uint(e.val))
               : "memory");
}
__device__ __forceinline__ bool ll_load(const ulonglong2* p, Pair* e, uint32_t epoch) {
  unsigned long long a, b;
  asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  e->idx = (int32_t)(uint32_t)a;
  e->val = __uint_as_float((uint32_t)b);
  return (uint32_t)(a >> 32) == epoch && (uint32_t)(b >> 32) == epoch;
}

// kPerThread: entries of a set per thread (k <= kPerThread * kPickThreads).
template <int kPerThread>
__global__ void __launch_bounds__(kPickThreads, 1)
k2_tree_small(const K2Rank* ranks, unsigned int rank_base, unsigned int P, unsigned int k, unsigned int kcap,
              unsigned int d, unsigned long long limit_ns) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmallShared& s = *reinterpret_cast<SmallShared*>(smem);
  uint32_t* const ent_idx = reinterpret_cast<uint32_t*>(smem + (sizeof(SmallShared) + 15) / 16 * 16);  // kEmpty: none
  const unsigned int half = (k + 3u) & ~3u;  // (keeps the table 16-byte aligned)
  float* const ent_val = reinterpret_cast<float*>(ent_idx + 2u * half);
  const unsigned int slots = small_slots(k);
  uint32_t* const words = reinterpret_cast<uint32_t*>(ent_val + 2u * half);
  const Table table{shared_address(words), slots, __clz(slots) + 1};
  const uint32_t bins_at = shared_address(s.hist);
  const unsigned int tid = threadIdx.x;
  const unsigned int me = rank_base + blockIdx.x;
  unsigned int* const bins = s.hist;

  // ---- before the predecessor has ended: the table
  auto clear_table = [&]() {
    for (unsigned int j = 4u * tid; j < slots; j += 4u * kPickThreads)
      *reinterpret_cast<uint4*>(&words[j]) = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
  };
  auto clear_bins = [&]() { reinterpret_cast<uint2*>(bins)[tid] = make_uint2(0u, 0u); };
  clear_table();
  clear_bins();
  if (tid == 0) {
    s.ok = 1;
    s.fresh_n = 0u;
    s.list_n = 0u;
    s.tie = 0u;
  }
  __syncthreads();
  pdl_begin(ranks);

  // the descriptor (several ranks' are put together by a kernel, possibly the one just before), then one round of loads
  const K2Rank& R = ranks[blockIdx.x];
  const Pair* const sel = R.sel;
  const unsigned int n_ahead = k < R.sel_cap ? k : R.sel_cap;
  const K1State* const st = R.st;
  unsigned int* const epoch_word = R.epoch;
  unsigned int* const result = R.n_global;
  Ctrl* const ctrl_pair = R.ctrl;
  float* const resid = R.resid;
  const unsigned int epoch = __ldcg(epoch_word);
  const unsigned int failed_before = __ldcg(&result[kResStatus]);
  const unsigned int heavy[2] = {__ldcg(&ctrl_pair[0].scratch[8]), __ldcg(&ctrl_pair[1].scratch[8])};
  unsigned int n_sel = __ldcg(&st->n_sel);
  uint32_t pred = __ldcg(reinterpret_cast<const unsigned int*>(&st->kth_mag)) & 0x7fffffffu;
  Pair own[kPerThread];
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    const unsigned int i = (unsigned int)u * kPickThreads + tid;
    own[u].idx = -1;
    own[u].val = 0.f;
    if (i < n_ahead) own[u] = ld_pair_cg(&sel[i]);
  }
  const unsigned int parity = epoch & 1u;
  Ctrl* const ctrl = ctrl_pair + parity;
  if (failed_before != 0u) {  // an earlier call failed: nothing is exchanged any more
    if (tid == 0) result[kResCount] = 0u;
    return;
  }
  if (n_sel > k) n_sel = k;
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    if ((unsigned int)u * kPickThreads + tid >= n_sel) own[u].idx = -1;
    else if ((unsigned int)own[u].idx >= d) {
      record_error(ctrl, ST_BOUNDS, 300);
      own[u].idx = -1;
    }
  }
  trace_stamp_of(ctrl, 0);
  // The other control block, for the next call: its header and stamps, and the histograms if the last call
  // took the form that uses them.
  {
    unsigned int* other = reinterpret_cast<unsigned int*>(ctrl_pair + (parity ^ 1u));
    const unsigned int n32 = (unsigned int)(heavy[parity ^ 1u] ? sizeof(Ctrl) : offsetof(Ctrl, hist)) / 4u;
    for (unsigned int i = tid; i < n32; i += kPickThreads) other[i] = 0u;
  }

  Pair nothing;
  nothing.idx = -1;
  nothing.val = 0.f;
  auto bin_of = [&](float v) {  // valid for magnitudes of at least pred
    const unsigned int b = (mag_key(v) - pred) >> kBandShift;
    return b < (unsigned int)kBins ? b : (unsigned int)kBins - 1u;
  };
  auto tally = [&](float v, unsigned int delta) {
    if (mag_key(v) >= pred) shared_add(bins_at + 4u * bin_of(v), delta);
  };
  // Entry e becomes number `at` of the union, or adds to the one of the same index.
  auto add = [&](Pair e, unsigned int at, unsigned int& fresh) {
    ent_idx[at] = kEmpty;
    if (e.idx < 0) return;
    const unsigned int have = table.enter((uint32_t)e.idx, at);
    if (have == at) {
      ent_idx[at] = (uint32_t)e.idx;
      ent_val[at] = e.val;
      tally(e.val, 1u);
      ++fresh;
    } else {
      const float old = ent_val[have], now = old + e.val;
      ent_val[have] = now;
      tally(old, 0xffffffffu);
      tally(now, 1u);
    }
  };
  auto count_fresh = [&](unsigned int fresh) {
    fresh = __reduce_add_sync(0xffffffffu, fresh);
    if (lane_id() == 0 && fresh) atomicAdd(&s.fresh_n, fresh);
  };
  // Receives up to k entries from `src` into e[] (idx -1: none at this place).  False after the limit.
  auto receive = [&](const ulonglong2* src, Pair (&e)[kPerThread], uint32_t where) {
    const uint64_t t0 = globaltimer_ns();
    unsigned int spins = 0;
    bool ok = s.ok != 0;
    unsigned int missing = 0;
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      e[u].idx = -1;
      e[u].val = 0.f;
      if ((unsigned int)u * kPickThreads + tid < k) missing |= 1u << u;
    }
    while (missing && ok) {
#pragma unroll
      for (int u = 0; u < kPerThread; ++u) {
        if (!(missing & (1u << u))) continue;
        Pair x;
        if (ll_load(&src[(unsigned int)u * kPickThreads + tid], &x, epoch)) {
          e[u] = x;
          missing &= ~(1u << u);
        }
      }
      if (missing && (++spins & 63u) == 0u) {
        if (aborted(ctrl)) {
          ok = false;
        } else if (globaltimer_ns() - t0 > limit_ns) {
          record_error(ctrl, ST_TIMEOUT_FLAG, where);
          ok = false;
        }
      }
    }
    if (!ok) s.ok = 0;
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      if (!ok || (missing & (1u << u))) e[u].idx = -1;
      else if (e[u].idx != -1 && (unsigned int)e[u].idx >= d) {
        record_error(ctrl, ST_BOUNDS, where + 10u);
        e[u].idx = -1;
      }
    }
  };
  // The k-th largest magnitude of the union (0 and no quota limit: all of at most k entries stay) and how many
  // entries equal to it stay.
  unsigned int quota = 0;
  auto threshold = [&]() -> uint32_t {
    if (s.fresh_n <= k) {
      quota = 0xffffffffu;
      return 0u;
    }
    uint2 counts = reinterpret_cast<const uint2*>(bins)[tid];
    Level lv{pred, 0x7fffffffu, kBandShift, true};
    unsigned int k_rem = k;
    for (bool direct = true;; direct = false) {
      if (find_bin(s, counts, k_rem) < k_rem) {  // the threshold lies below the predicted band: entries cancelled
        lv = Level{0u, 0x7fffffffu, 20u, false};
        direct = false;
      } else {
        k_rem = s.res_krem;
        if (!lv.narrow(s.res_bin)) break;
      }
      if (direct) {  // few entries in the bin: rank them, every warp for itself
        for (unsigned int j = tid; j < 2u * k; j += kPickThreads) {
          const uint32_t key = mag_key(ent_val[j]);
          if (ent_idx[j] != kEmpty && lv.has(key)) {
            const unsigned int at = atomicAdd(&s.list_n, 1u);
            if (at < kRankList) s.list[at] = key;
          }
        }
        __syncthreads();
        const unsigned int n = s.list_n;
        if (n <= kRankList) {
          const uint32_t key = lane_id() < n ? s.list[lane_id()] : 0u;
          unsigned int above = 0, equal = 0;
          for (unsigned int q = 0; q < n; ++q) {
            const uint32_t other = s.list[q];
            above += other > key ? 1u : 0u;
            equal += other == key ? 1u : 0u;
          }
          const bool is = lane_id() < n && above < k_rem && k_rem <= above + equal;
          const int who = __ffs(__ballot_sync(0xffffffffu, is)) - 1;
          quota = k_rem - __shfl_sync(0xffffffffu, above, who);
          return __shfl_sync(0xffffffffu, key, who);
        }
      }
      clear_bins();
      __syncthreads();
      for (unsigned int j = tid; j < 2u * k; j += kPickThreads) {
        const uint32_t key = mag_key(ent_val[j]);
        if (ent_idx[j] != kEmpty && lv.has(key)) shared_add(bins_at + 4u * lv.bin(key), 1u);
      }
      __syncthreads();
      counts = reinterpret_cast<const uint2*>(bins)[tid];
    }
    quota = k_rem;
    return lv.lo;
  };
  // Keeps what reaches the threshold: out(position, entry) for each, positions 0, 1, ...; a warp's entries of one
  // trip side by side.  Returns how many.  Entries leave the shared arrays before anything is put out, so out
  // may write there.
  auto keep_largest = [&](uint32_t th, auto out) {
    Pair e[2 * kPerThread];
    unsigned int won = 0, n = 0;
#pragma unroll
    for (int u = 0; u < 2 * kPerThread; ++u) {
      const unsigned int j = (unsigned int)u * kPickThreads + tid;
      e[u] = nothing;
      if ((unsigned int)u * kPickThreads >= 2u * k) continue;  // uniform
      if (j < 2u * k && ent_idx[j] != kEmpty) {
        e[u].idx = (int32_t)ent_idx[j];
        e[u].val = ent_val[j];
      }
      const bool stays = passes(e[u].idx >= 0, mag_key(e[u].val), th, quota, &s.tie);
      if (stays) won |= 1u << u;
      else if (e[u].idx >= 0) ent_idx[j] = kEmpty;  // (a look-up of its index finds no entry any more)
      n += (unsigned int)__popc(__ballot_sync(0xffffffffu, stays));
    }
    const int w = (int)(tid >> 5);
    if (lane_id() == 0) s.warp_n[0][w] = n;
    __syncthreads();
    const unsigned int theirs = s.warp_n[0][lane_id()];
    unsigned int pos = __reduce_add_sync(0xffffffffu, (int)lane_id() < w ? theirs : 0u);
    const unsigned int total = __reduce_add_sync(0xffffffffu, theirs);
#pragma unroll
    for (int u = 0; u < 2 * kPerThread; ++u) {
      if ((unsigned int)u * kPickThreads >= 2u * k) continue;
      const bool stays = (won & (1u << u)) != 0u;
      const unsigned int m = __ballot_sync(0xffffffffu, stays);
      if (stays) out(pos + __popc(m & lanemask_lt()), e[u]);
      pos += (unsigned int)__popc(m);
    }
    return total;
  };

  Pair* const G = R.gout + (size_t)parity * kcap;
  unsigned int n_g = 0;
  unsigned int rounds = 0;
  while ((1u << rounds) < P) ++rounds;
  if (me & 1u) {
    // ---- sender of round 0: the selection as it is (places without an entry carry index -1)
    ulonglong2* dst = R.peer_ll[me - 1u] + ll_off(parity, 0);
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      const unsigned int i = (unsigned int)u * kPickThreads + tid;
      if (i < k) ll_store(&dst[i], own[u].idx >= 0 ? own[u] : nothing, epoch);
    }
    trace_stamp_of(ctrl, 1 + 6);
    trace_stamp_of(ctrl, 1 + 7);
  } else {
    unsigned int fresh = 0;
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      const unsigned int i = (unsigned int)u * kPickThreads + tid;
      if (i < k) add(own[u], i, fresh);
    }
    count_fresh(fresh);
    for (unsigned int r = 0; r < rounds; ++r) {
      const unsigned int bit = 1u << r;
      trace_stamp_of(ctrl, 1 + 8 * r + 0);
      Pair e[kPerThread];
      receive(R.ll + ll_off(parity, r), e, 210 + r);
      trace_stamp_of(ctrl, 1 + 8 * r + 1);
      __syncthreads();  // this rank's entries are in the table
      trace_stamp_of(ctrl, 1 + 8 * r + 2);
      fresh = 0;
#pragma unroll
      for (int u = 0; u < kPerThread; ++u) {
        const unsigned int i = (unsigned int)u * kPickThreads + tid;
        if (i < k) add(e[u], k + i, fresh);
      }
      count_fresh(fresh);
      __syncthreads();
      trace_stamp_of(ctrl, 1 + 8 * r + 3);
      const uint32_t th = threshold();
      trace_stamp_of(ctrl, 1 + 8 * r + 4);
      if (r + 1 == rounds) {  // rank 0: the global set goes to every rank
        n_g = keep_largest(th, [&](unsigned int at, Pair x) {
          if (!s.ok) return;
          for (unsigned int q = 1; q < P; ++q) ll_store(R.peer_ll[q] + ll_off(parity, kMaxRounds) + at, x, epoch);
          st_pair(&G[at], x);
        });
        for (unsigned int i = n_g + tid; i < k && s.ok; i += kPickThreads)
          for (unsigned int q = 1; q < P; ++q) ll_store(R.peer_ll[q] + ll_off(parity, kMaxRounds) + i, nothing, epoch);
        trace_stamp_of(ctrl, 1 + 8 * r + 5);
      } else if ((me & (4u * bit - 1u)) == 2u * bit) {  // sender of the next round: leaves the tree
        ulonglong2* dst = R.peer_ll[me - 2u * bit] + ll_off(parity, r + 1);
        const unsigned int n = keep_largest(th, [&](unsigned int at, Pair x) {
          if (s.ok) ll_store(&dst[at], x, epoch);
        });
        for (unsigned int i = n + tid; i < k && s.ok; i += kPickThreads) ll_store(&dst[i], nothing, epoch);
        trace_stamp_of(ctrl, 1 + 8 * r + 5);
        trace_stamp_of(ctrl, 1 + 8 * (r + 1) + 7);
        break;
      } else {  // receiver again: the set moves to the front, with a new table and bins above the new threshold
        clear_table();
        clear_bins();
        const uint32_t next_pred = th ? th : pred;
        const unsigned int n = keep_largest(th, [&](unsigned int at, Pair x) {  // (its barrier: all is cleared)
          ent_idx[at] = (uint32_t)x.idx;
          ent_val[at] = x.val;
          table.enter((uint32_t)x.idx, at);
          if (mag_key(x.val) >= next_pred) {
            const unsigned int b = (mag_key(x.val) - next_pred) >> kBandShift;
            shared_add(bins_at + 4u * (b < (unsigned int)kBins ? b : (unsigned int)kBins - 1u), 1u);
          }
        });
        pred = next_pred;
        for (unsigned int i = n + tid; i < k; i += kPickThreads) ent_idx[i] = kEmpty;
        if (tid == 0) {
          s.fresh_n = n;
          s.list_n = 0u;
          s.tie = 0u;
        }
        trace_stamp_of(ctrl, 1 + 8 * r + 5);
      }
    }
  }

  // ---- the global set: rank 0 has sent it to every rank; the others put it into their buffer
  float back[kPerThread];  // residual at the own entries: most of them get their value back
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    back[u] = 0.f;
    if (own[u].idx >= 0) back[u] = resid[own[u].idx];
  }
  if (me == 0u) {
    trace_stamp_of(ctrl, 40);
    __syncthreads();  // the losers are out of the arrays
  } else {
    // While the root merges, the table over the own selection; what arrives strikes its index off there.  (A table
    // over the global set is entered and looked up after the last entry is there: 0.9 us more from its arrival to
    // the end, k = 1 000; whole call with two ranks 12.3 -> 11.4 us, eight 26.2 -> 25.1, k = 2 000 18.3 -> 17.1.)
    __syncthreads();
    clear_table();
    if (tid == 0) s.fresh_n = 0u;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      const unsigned int at = (unsigned int)u * kPickThreads + tid;
      if (own[u].idx < 0) continue;
      table.enter((uint32_t)own[u].idx, at);
      ent_idx[at] = (uint32_t)own[u].idx;
    }
    __syncthreads();
    Pair e[kPerThread];
    receive(R.ll + ll_off(parity, kMaxRounds), e, 410);
    trace_stamp_of(ctrl, 40);
    unsigned int n = 0;
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      if (e[u].idx < 0) continue;  // (those without an entry are the last ones)
      st_pair(&G[(unsigned int)u * kPickThreads + tid], e[u]);
      const unsigned int at = table.find((uint32_t)e[u].idx);
      if (at != kEmpty) ent_idx[at] = kEmpty;
      ++n;
    }
    count_fresh(n);
    __syncthreads();
    n_g = s.fresh_n;
  }
  trace_stamp_of(ctrl, 41);
  // ---- residual put-back of S_local \ S_global
  if (s.ok) {
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      if (own[u].idx < 0) continue;
      bool lost;
      if (me == 0u) {
        const unsigned int at = table.find((uint32_t)own[u].idx);
        lost = at == kEmpty || ent_idx[at] != (uint32_t)own[u].idx;
      } else {
        lost = ent_idx[(unsigned int)u * kPickThreads + tid] != kEmpty;
      }
      if (lost) resid[own[u].idx] = back[u] + own[u].val;
    }
  }
  trace_stamp_of(ctrl, 42);
  __syncthreads();
  if (tid != 0) return;
  if (aborted(ctrl)) {
    result[kResCount] = 0u;
    const unsigned int status = ld_relaxed_gpu_u32(&ctrl->status);
    if (atomicCAS(&result[kResStatus], 0u, status ? status : (unsigned int)ST_TIMEOUT_FLAG) == 0u) {
      result[kResWhere] = ld_relaxed_gpu_u32(&ctrl->where);
      result[kResEpoch] = epoch;
    }
  } else {
    result[kResCount] = n_g;
    *epoch_word = epoch + 1u;
  }
}

bool k2_small_serves(unsigned int nranks, unsigned int k, unsigned int nctas) {
  return nctas == 1 && k <= kLLMaxK && nranks <= 8u;  // 8: the portable cluster size
}

int k2_small_launch(const K2Rank* ranks, unsigned int nranks, unsigned int rank_base, unsigned int P, unsigned int k,
                    unsigned int kcap, unsigned int d, unsigned long long limit_ns, cudaStream_t stream) {
  static std::atomic<int> ready[64];  // per device
  const DeviceInfo* di = gtk_device_info();
  if (!di || di->device < 0 || di->device >= 64) return GTK_ERR_CUDA;
  if (!ready[di->device].load(std::memory_order_relaxed)) {
    for (auto f : {k2_tree_small<1>, k2_tree_small<2>})
      if (cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)small_smem_bytes(kLLMaxK)) != cudaSuccess)
        return GTK_ERR_CUDA;
    ready[di->device].store(1, std::memory_order_relaxed);
  }
  const auto fn = k <= kPickThreads ? k2_tree_small<1> : k2_tree_small<2>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nranks);
  cfg.blockDim = dim3(kPickThreads);
  cfg.dynamicSmemBytes = small_smem_bytes(k);
  cfg.stream = stream;
  // Emulated ranks wait for one another: as one cluster they are scheduled together.
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = nranks;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = nranks > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, ranks, rank_base, P, k, kcap, d, limit_ns);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}

}  // namespace gtk
