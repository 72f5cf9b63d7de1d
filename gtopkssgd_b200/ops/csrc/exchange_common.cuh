// Device-side pieces shared by the two sparse exchange kernels (K2: gTop-k tree,
// K2t: Top-k all-gather): the per-rank descriptor, the wire words, flags, the
// direct-address merge of two sparse sets, and the residual put-back.
//
// Merging without sorting: each rank owns an int32 table `map` of d entries.
// To join set A (n_a entries) with set B, A first writes map[A[i].idx] = i; an
// entry (j, v) of B is shared iff p = map[j] satisfies p < n_a && A[p].idx == j.
// The second test makes stale table contents harmless, so the table is never
// cleared.
#pragma once
#include "select_common.cuh"
#include "host_api.h"

namespace gtk {

// Layout of the symmetric (peer-visible) region of one rank, identical on all
// ranks.  Two parities (epoch & 1) so that a fast sender of call e+1 never
// overwrites what a slow reader of call e still needs.
//   slots : [2][kMaxRounds + 1][kcap] wire words   receive slot of each tree round and of the broadcast
//   ag    : [2][kMaxPeers][kcap] pairs    all-gather slots, one per source rank (K2t only)
//   wire  : [2][kMaxPeers][kcap] wire words   the same for the re-selecting form (K2t only)
//   gout  : [2][kcap] pairs               the global top-k set
//   flags : [2][kFlagsPerParity] u64      (epoch << 32) | count
//   ll    : [2][kMaxRounds + 1][kLLMaxK] 16-byte entries with their epoch (k2_tree_small.cu); the last
//           row of a parity is the broadcast's
constexpr int kFlagBcast = kMaxRounds;             // flag index of the broadcast
constexpr int kFlagAg0 = kMaxRounds + 1;           // first all-gather flag (one per source)
constexpr int kFlagsPerParity = kMaxRounds + 1 + kMaxPeers;
constexpr unsigned int kLLMaxK = 2048;  // largest k of the small tree exchange (k2_tree_small.cu)
__host__ __device__ constexpr size_t ll_off(unsigned int parity, unsigned int round) {
  return ((size_t)parity * (kMaxRounds + 1) + round) * kLLMaxK;
}

struct K2Rank {
  const Pair* sel;        // local selection written by K1
  unsigned int sel_cap;   // pairs that its buffer holds
  const K1State* st;      // st->n_sel = number of local pairs
  // Merge buffers.  Tree: [kcap] and [2 * kcap] pairs, the second half of work[1] for received entries.  K2t:
  // work[0] is the union [work_cap], work[1] holds a word per entry of it.
  Pair* work[2];
  int32_t* map;           // [d] direct-address table
  float* resid;           // [d] residual
  unsigned long long* slots;  // local symmetric buffers
  Pair* ag;
  unsigned long long* wire;
  Pair* gout;
  uint64_t* flags;
  ulonglong2* ll;
  Ctrl* ctrl;             // TWO control blocks: call e uses block (e & 1) and cleans the other one itself
  unsigned int* n_global; // kResWords device words: result of the last call, see kRes* below
  unsigned int* epoch;    // device word: call counter (starts at 1); the kernel reads it at entry and
                          // adds one after its last barrier, so a replayed CUDA graph needs no new argument
  unsigned long long* peer_slots[kMaxPeers];
  Pair* peer_ag[kMaxPeers];
  unsigned long long* peer_wire[kMaxPeers];
  uint64_t* peer_flags[kMaxPeers];
  ulonglong2* peer_ll[kMaxPeers];
};

// The tree exchange for small sets (k2_tree_small.cu).
bool k2_small_serves(unsigned int nranks, unsigned int k, unsigned int nctas);
int k2_small_launch(const K2Rank* ranks, unsigned int nranks, unsigned int rank_base, unsigned int P, unsigned int k,
                    unsigned int kcap, unsigned int d, unsigned long long limit_ns, cudaStream_t stream);

// Result words of an exchange (K2Rank::n_global).  kResCount is what the consumer (K3) reads: the
// number of pairs in gout[parity], 0 after a failed call.  The other three are written once, by
// the first failing call, and never cleared by a kernel: while kResStatus is non-zero every later
// call returns at once with an empty result.
constexpr int kResCount = 0;
constexpr int kResStatus = 1;
constexpr int kResWhere = 2;
constexpr int kResEpoch = 3;
constexpr int kResWords = 4;

struct ExchangeShared {
  SelectShared sel;
  unsigned int payload;
  int ok;
};

__device__ __forceinline__ size_t slot_off(unsigned int parity, unsigned int round,
                                           unsigned int kcap) {
  return ((size_t)parity * (kMaxRounds + 1) + round) * kcap;
}

// The wire word of a slot: one pair in one 8-byte store that no reader sees half of, never 0 (an index has its
// top bit clear, on the wire set), so that a word that has been cleared says whether its pair has arrived.  A
// receiver polls the words themselves and clears what it has taken: a set crosses without a system-wide fence
// in every CTA that stored, a barrier over them and a flag's release behind it, which took 6 us per hop.  The
// slot's next use is two calls later, which its sender starts only after this receiver took part in the call
// between (its set is in the one that the root sent round).
__device__ __forceinline__ void wire_store(unsigned long long* slot, Pair e) {
  e.idx ^= (int32_t)0x80000000;
  st_relaxed_sys_u64(slot, pair_bits(e));
}
// Brings the table's line for idx into L2, ahead of a look-up behind a barrier.  Tables of up to 2 M entries (8 MB a
// rank) are there anyway: eight ranks of 4 M entries 95.0 -> 91.1 us ('topk2'), of 1 M 41.0 -> 42.1 without the rule.
__device__ __forceinline__ void prefetch_entry(const int32_t* map, int32_t idx, unsigned int d) {
  if (d > 2000000u && idx >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(&map[idx]));
}

// Receives the words slot + at(j) of this thread, for the j of `want`, into e[j] (idx -1: not wanted, or an index
// outside [0, d)) and clears them.  Returns false, the error recorded, when the limit runs out or the rank gives up.
template <int N, typename At>
__device__ __forceinline__ bool wire_receive(unsigned long long* slot, unsigned int want, At at, Pair (&e)[N],
                                             unsigned int d, Ctrl* ctrl, uint64_t limit_ns, uint32_t where) {
  const uint64_t t0 = want ? globaltimer_ns() : 0ull;
  unsigned int spins = 0;
  while (want) {
    unsigned long long w[N];
#pragma unroll
    for (int j = 0; j < N; ++j) w[j] = (want & (1u << j)) ? ld_relaxed_sys_u64(slot + at(j)) : 0ull;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (w[j] == 0ull) continue;
      slot[at(j)] = 0ull;
      want &= ~(1u << j);
      e[j] = bits_pair(w[j]);
      e[j].idx ^= (int32_t)0x80000000;
      if ((unsigned int)e[j].idx >= d) {
        record_error(ctrl, ST_BOUNDS, where + 90u);
        e[j].idx = -1;
      }
    }
    if (want && (++spins & 63u) == 0u) {
      if (aborted(ctrl)) return false;
      if (globaltimer_ns() - t0 > limit_ns) {
        record_error(ctrl, ST_TIMEOUT_FLAG, where);
        return false;
      }
    }
  }
  return true;
}
__device__ __forceinline__ size_t ag_off(unsigned int parity, unsigned int src, unsigned int kcap) {
  return ((size_t)parity * kMaxPeers + src) * kcap;
}
__device__ __forceinline__ size_t flag_off(unsigned int parity, unsigned int which) {
  return (size_t)parity * kFlagsPerParity + which;
}

// Calls f(pair, i) for this thread's entries of a list, with the loads of four of them in flight.
template <typename F>
__device__ __forceinline__ void for_pairs(const Pair* list, unsigned int n, unsigned int lane0, unsigned int stride, F f) {
  constexpr int N = 4;
  for (unsigned int i0 = lane0; i0 < n; i0 += N * stride) {
    Pair e[N];
#pragma unroll
    for (int t = 0; t < N; ++t)
      if (i0 + t * stride < n) e[t] = ld_pair_cg(&list[i0 + t * stride]);
#pragma unroll
    for (int t = 0; t < N; ++t)
      if (i0 + t * stride < n) f(e[t], i0 + t * stride);
  }
}

// Called by all threads of a CTA of a multi-CTA rank after its last store into peer memory of a phase
// and before the rank's barrier: one thread issues a system-scope fence on behalf of the CTA (the
// __syncthreads orders the other threads' stores before it).  By the PTX memory model the flag's own
// st.release.sys, issued after the rank's barrier, already covers these stores (the barrier is a
// morally strong synchronisation and release is cumulative); the fence makes each SM wait for the
// acknowledgement of its own NVLink stores instead of leaving that to one SM's release on behalf of
// all, which is the form library collectives use (one fencing thread per CTA that stored).  A rank
// served by a single CTA needs no extra fence: the thread that raises the flag sits in the CTA that
// stored.  Cost: 2-3 us per sending phase.
__device__ __forceinline__ void cta_fence_peer_stores(bool single_cta) {
  if (single_cta) return;
  __syncthreads();
  if (threadIdx.x == 0) __threadfence_system();
}

// Publish: st.release.sys orders every store that happens-before it (this
// thread's own and, through the preceding barrier, every other thread's).
__device__ __forceinline__ void release_flag(uint64_t* flag, uint32_t epoch, uint32_t count) {
  st_release_sys_u64(flag, ((uint64_t)epoch << 32) | (uint64_t)count);
}

// One thread per CTA waits for the flag, the CTA learns the count.
__device__ __forceinline__ bool cta_wait_flag(ExchangeShared& sh, const uint64_t* flag,
                                              uint32_t epoch, Ctrl* ctrl, uint64_t limit_ns,
                                              uint32_t where, unsigned int* count) {
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t payload = 0;
    sh.ok = wait_flag(flag, epoch, ctrl, limit_ns, where, &payload) ? 1 : 0;
    sh.payload = payload;
  }
  __syncthreads();
  *count = sh.payload;
  return sh.ok != 0;
}

// Residual put-back (compression.py:66-75 in the reference): every locally
// selected entry whose index is not in the global set returns to the residual.
// Requires map[] built over G.
__device__ __forceinline__ void put_back(const Pair* sel, unsigned int n_sel, const Pair* G,
                                         unsigned int n_g, const int32_t* map, float* resid,
                                         unsigned int d, unsigned int cta, unsigned int nct) {
  const unsigned int stride = nct * kSelThreads;
  constexpr int N = 4;  // entries per thread whose four dependent loads go together
  for (unsigned int i0 = cta * kSelThreads + threadIdx.x; i0 < n_sel; i0 += N * stride) {
    Pair e[N];
    unsigned int p[N];
    float back[N];
#pragma unroll
    for (int t = 0; t < N; ++t) {
      e[t].idx = -1;
      e[t].val = 0.f;
      if (i0 + t * stride < n_sel) e[t] = sel[i0 + t * stride];
      if ((unsigned int)e[t].idx >= d) e[t].idx = -1;
    }
#pragma unroll
    for (int t = 0; t < N; ++t) p[t] = e[t].idx >= 0 ? (unsigned int)__ldcg(&map[e[t].idx]) : 0xffffffffu;
#pragma unroll
    for (int t = 0; t < N; ++t)
      if (p[t] < n_g && ld_pair_cg(&G[p[t]]).idx == e[t].idx) e[t].idx = -1;
#pragma unroll
    for (int t = 0; t < N; ++t) back[t] = e[t].idx >= 0 ? resid[e[t].idx] + e[t].val : 0.f;
#pragma unroll
    for (int t = 0; t < N; ++t)
      if (e[t].idx >= 0) resid[e[t].idx] = back[t];
  }
}

}  // namespace gtk
