// K2: the gTop-k recursive-doubling exchange as one persistent kernel.
//
// Semantics of gtopk_sparse_allreduce in the reference (allreducer.py:71-163):
// log2(P) rounds; in round r rank i + 2^r sends its k pairs to rank i for every
// i = 0 (mod 2^(r+1)); the receiver sums values on shared indices and keeps the k
// largest magnitudes of the union; rank 0 ends with the global set and
// broadcasts it; every rank returns "selected locally but not globally" values
// to its residual (compression.py:66-75).
//
// Here every transfer is an NVLink peer store into the partner's receive slot,
// one 8-byte word per pair that says by itself whether it has arrived; an
// epoch-stamped word in the partner's memory says how many to expect.  A
// receiver polls only its own memory.  No MPI, no NCCL, no host staging, no
// per-round barrier between ranks, no fence between data and flag.
//
// One launch serves gridDim.y ranks: 1 in production (one process per GPU), P
// when all ranks are emulated on one GPU for testing, in which case the launch
// is cooperative so that all CTAs are co-resident and the flag waits make
// progress.  gridDim.x CTAs serve each rank and meet in RankBarrier.
//
// A merged set is compacted straight to where the next phase reads it: into the
// partner's receive slot when this rank sends in the next round, into every
// rank's broadcast slot after the last round (rank 0), into the local work
// buffer otherwise.  So only round 0 has a separate push, and there is no
// separate broadcast copy.
//
// What bounds it: a chain of phases of 2 to 6 us, each a round of L2 or scattered
// DRAM accesses (the table spans d) and a barrier; past k of about 200 000 the
// scattered accesses themselves (45 a ns).  Two ranks, k = 66 034, the same
// selection exchanged again and again: 40 us with flags behind fenced plain stores
// and the put-back at the end, 23 us now (k = 255 570: 88 and 70; four ranks, k =
// 14 728: 43 and 32; eight ranks, k = 40 000: 122 and 85).
//
// No host-side clearing: the rank owns two control blocks; call e uses block
// (e & 1) and zeroes the other one for call e + 1 at its beginning, where the stores
// are gone long before anything waits for them.
//
// Failure: any wait that runs out, any capacity or bounds error makes the call
// publish an EMPTY global set (n_global = 0, so the consumer applies nothing) and
// a sticky status in the result words; the call counter is not advanced and every
// later call returns at once with an empty set until the host has rebuilt the
// exchange.  A rank that has put its selection back by then keeps it in the
// residual, as an empty global set asks for.
#include <cstddef>
#include "exchange_common.cuh"

namespace gtk {

// Union entries that each thread keeps in registers across the phases of a round.  The default CTA counts leave
// 2 to 4 per thread up to k of about 150 000; the rest is read again from memory, as many at a time.
constexpr int kK2Cache = 4;
// Entries of the own selection that each thread reads with the descriptor's first words, an L2 round trip (0.8 us)
// before it knows how many there are.  The default CTA counts leave at most two up to k of 150 000 where the GPU has one
// or two ranks, 75 000 with four and 37 000 with eight; further ones (9 for eight ranks of 170 000) come behind, four
// loads at a time.  With the control block cleared at the
// beginning and old residual values kept beside their indices (one look-up less behind an arrival): three worlds of two
// ranks and k = 66 034 in turn, with the update, 39.1 -> 37.75 us; four of k = 16 000 37.8 -> 37.1.
constexpr int kK2Own = 2;

struct K2Shared {
  ExchangeShared ex;
  unsigned int band[kHistBins];   // this CTA's share of the first selection level, counted on the fly
};

__device__ __forceinline__ void band_clear(K2Shared& sh) {
  for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) sh.band[i] = 0u;
  __syncthreads();
}
// Adds this CTA's (possibly "negative", i.e. wrapped) partial counts to a round's global ones and zeroes the
// shared copy.
__device__ __forceinline__ void band_flush(K2Shared& sh, unsigned int* ghist) {
  __syncthreads();
  for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) {
    const unsigned int c = sh.band[i];
    if (c) atomicAdd(&ghist[i], c);
    sh.band[i] = 0u;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kSelThreads, 2)
k2_gtopk_exchange(const K2Rank* __restrict__ ranks, unsigned int rank_base, unsigned int P,
                  unsigned int k, unsigned int kcap, unsigned int d, unsigned long long limit_ns,
                  int use_cluster) {
  __shared__ K2Shared sh;
  SelectShared& ss = sh.ex.sel;
  const K2Rank& R = ranks[blockIdx.y];
  // One round of loads (a load behind the check of the status would be another round trip).
  const unsigned int epoch = __ldcg(R.epoch);  // every CTA reads it before its first barrier
  const unsigned int status = __ldcg(&R.n_global[kResStatus]);
  unsigned int n_sel = __ldcg(&R.st->n_sel);
  const float kth_mag = __ldcg(&R.st->kth_mag);
  const unsigned int me = rank_base + blockIdx.y;
  const unsigned int cta = blockIdx.x, nct = gridDim.x;
  const unsigned int stride = nct * kSelThreads;
  const unsigned int lane0 = cta * kSelThreads + threadIdx.x;  // union index of this thread's trip 0
  const unsigned int n_ahead = k < R.sel_cap ? k : R.sel_cap;
  Pair own[kK2Own];  // this thread's first entries of the selection (beyond n_sel: whatever is there, never looked at)
#pragma unroll
  for (int t = 0; t < kK2Own; ++t) {
    own[t].idx = -1;
    own[t].val = 0.f;
    if (lane0 + t * stride < n_ahead) own[t] = ld_pair_cg(&R.sel[lane0 + t * stride]);
  }
  const unsigned int parity = epoch & 1u;
  Ctrl* ctrl = R.ctrl + parity;
  int32_t* const map = R.map;
  RankBarrier bar{ctrl, nct, 0u, limit_ns, use_cluster != 0};
  // Says how many pairs a slot of rank q gets; they follow, or have come already, in no order.
  auto announce = [&](unsigned int q, unsigned int which, unsigned int n) {
    st_relaxed_sys_u64(reinterpret_cast<unsigned long long*>(R.peer_flags[q] + flag_off(parity, which)),
                       ((unsigned long long)epoch << 32) | n);
  };
  // Calls f(entry, i) for this thread's entries of the own selection; behind the ones read ahead, four loads in flight.
  auto for_own = [&](auto f) {
#pragma unroll
    for (int t = 0; t < kK2Own; ++t) {
      const unsigned int i = lane0 + t * stride;
      if (i < n_sel) f(i < n_ahead ? own[t] : ld_pair_cg(&R.sel[i]), i);
    }
    for_pairs(R.sel, n_sel, lane0 + kK2Own * stride, stride, f);
  };
  // Leaves an empty result and the sticky status behind; called by every CTA that gives up.
  auto fail = [&]() {
    if (threadIdx.x == 0) {
      atomicExch(&R.n_global[kResCount], 0u);
      unsigned int st = ld_relaxed_gpu_u32(&ctrl->status);
      if (st == 0u) st = ST_TIMEOUT_BARRIER;  // left because another CTA of the rank did
      if (atomicCAS(&R.n_global[kResStatus], 0u, st) == 0u) {
        R.n_global[kResWhere] = ld_relaxed_gpu_u32(&ctrl->where);
        R.n_global[kResEpoch] = epoch;
      }
    }
  };
  if (status != 0u) {  // an earlier call failed: nothing is exchanged any more
    if (cta == 0 && threadIdx.x == 0) R.n_global[kResCount] = 0u;
    return;
  }

  if (n_sel > kcap) n_sel = kcap;
  unsigned int rounds = 0;
  while ((1u << rounds) < P) ++rounds;
  band_clear(sh);
  if (cta == 0 && threadIdx.x == 0) ctrl->scratch[8] = 1u;  // this block's histograms will need clearing
  // The other control block, for the next call (its last user was the call before).
  {
    uint4* other = reinterpret_cast<uint4*>(R.ctrl + (parity ^ 1u));
    const size_t nvec16 = (offsetof(Ctrl, hist) + (size_t)(rounds + 1) * sizeof(((Ctrl*)0)->hist[0])) / 16;
    for (size_t i = lane0; i < nvec16; i += stride) other[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  trace_stamp(ctrl, 0);
  // Every live entry of a round's union is counted once in the band above `pred` (delta = 1 adds, 0xffffffff
  // removes).  A prediction: for gradient tails the union's k-th magnitude is a few per cent above this rank's own,
  // but where entries of opposite sign cancel it is below, at any distance (bin 0; the counting sweeps then).
  uint32_t pred = mag_key(kth_mag);  // round 0: K1's k-th magnitude, then the previous round's threshold
  auto tally = [&](float v, unsigned int delta) { atomicAdd(&sh.band[band_bin(mag_key(v), pred)], delta); };

  if (me & 1u) {
    // ---- sender of round 0: push the selection into the partner's slot
    if (cta == 0 && threadIdx.x == 0) announce(me - 1u, 0, n_sel);
    unsigned long long* const dst = R.peer_slots[me - 1u] + slot_off(parity, 0, kcap);
    for_own([&](Pair e, unsigned int i) { wire_store(&dst[i], e); });
    trace_stamp(ctrl, 1 + 6);
    trace_stamp(ctrl, 1 + 7);
  } else {
    // ---- receiver.  A = current set in a writable work buffer, with map[] and the band counts
    // describing it (built here before round 0, by the previous compaction afterwards).
    for_own([&](Pair e, unsigned int i) {
      if ((unsigned int)e.idx < d) {
        map[e.idx] = (int32_t)i;
        tally(e.val, 1u);
      } else {
        record_error(ctrl, ST_BOUNDS, 300);
        e.idx = -1;
      }
      st_pair(&R.work[0][i], e);
    });
    bar.arrive();
  }
  unsigned int n_cur = n_sel;
  int cur_buf = 0;  // of the two work buffers
  for (unsigned int r = 0; (me & 1u) == 0u && r < rounds; ++r) {
    const unsigned int bit = 1u << r;
    const bool copied = r == 0u;
    Pair* const A = R.work[cur_buf];
    unsigned int n_b = 0;
    trace_stamp(ctrl, 1 + 8 * r + 0);
    if (!cta_wait_flag(sh.ex, R.flags + flag_off(parity, r), epoch, ctrl, limit_ns, 210 + r, &n_b)) {
      fail();
      return;
    }
    trace_stamp(ctrl, 1 + 8 * r + 1);
    if (n_b > kcap) {
      record_error(ctrl, ST_CAPACITY, 220 + r);
      n_b = kcap;
    }
    unsigned long long* const slot = R.slots + slot_off(parity, r, kcap);
    Pair* const B = R.work[1] + kcap;  // what is received beyond the register cache
    const unsigned int n_a = n_cur;
    const unsigned int n_u = n_a + n_b;
    const unsigned int trips = (n_u + stride - 1) / stride;

    // ---- probe: every thread takes its B entries off the slot, joins them against A (sum on shared
    // indices) and keeps them in registers; three dependent loads, issued level by level.
    auto receive = [&](Pair (&e)[kK2Cache], unsigned int t0) {
      unsigned int want = 0;
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        const unsigned int i = (t0 + t) * stride + lane0;
        e[t].idx = -1;
        e[t].val = 0.f;
        if (t0 + t < trips && i >= n_a && i < n_u) want |= 1u << t;
      }
      return wire_receive(slot, want, [&](int t) { return (size_t)((t0 + t) * stride + lane0 - n_a); }, e, d, ctrl,
                          limit_ns, 212 + r);
    };
    auto join = [&](Pair (&e)[kK2Cache]) {
      unsigned int pm[kK2Cache];
      Pair a[kK2Cache];
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        pm[t] = 0xffffffffu;
        if (e[t].idx >= 0) pm[t] = (unsigned int)__ldcg(&map[e[t].idx]);
      }
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        a[t].idx = -1;
        if (pm[t] < n_a) a[t] = ld_pair_cg(&A[pm[t]]);
      }
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        if (e[t].idx < 0) continue;
        if (a[t].idx == e[t].idx) {
          const float nv = a[t].val + e[t].val;
          A[pm[t]].val = nv;  // A[p] belongs to another thread's sweep: goes through memory
          tally(a[t].val, 0xffffffffu);
          tally(nv, 1u);
          e[t].idx = -1;
        } else {
          tally(e[t].val, 1u);
        }
      }
    };
    Pair c[kK2Cache];
    bool ok = receive(c, 0);
#pragma unroll
    for (int t = 0; t < kK2Cache; ++t) prefetch_entry(map, c[t].idx, d);
    // A and map must be complete: after the copy above that needs a barrier, after a previous
    // round its closing barrier already gave it
    if (!__syncthreads_and(ok) || (copied && !bar.wait(230 + r))) { fail(); return; }
    trace_stamp(ctrl, 1 + 8 * r + 2);
    join(c);
    for (unsigned int t0 = kK2Cache; t0 < trips && ok; t0 += kK2Cache) {
      Pair e[kK2Cache];
      ok = receive(e, t0);
      join(e);
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        const unsigned int i = (t0 + t) * stride + lane0;
        if (t0 + t < trips && i >= n_a && i < n_u) st_pair(&B[i - n_a], e[t]);
      }
    }
    if (!__syncthreads_and(ok)) { fail(); return; }
    band_flush(sh, ctrl->hist[r][0]);
    if (!bar.sync(240 + r)) { fail(); return; }  // sums and the on-the-fly histograms complete
    trace_stamp(ctrl, 1 + 8 * r + 3);

    // ---- every thread now loads its A entries (with the merged values) next to its B entries
#pragma unroll
    for (int t = 0; t < kK2Cache; ++t) {
      const unsigned int i = (unsigned int)t * stride + lane0;
      if ((unsigned int)t < trips && i < n_a) c[t] = ld_pair_cg(&A[i]);
    }
    auto entry = [&](unsigned int t) -> Pair {  // entry of trip t >= kK2Cache, from memory
      const unsigned int i = t * stride + lane0;
      Pair e;
      e.idx = -1;
      e.val = 0.f;
      if (i < n_u) e = ld_pair_cg(i < n_a ? &A[i] : &B[i - n_a]);
      return e;
    };

    // ---- re-select
    auto visit = [&](auto f) {
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t)
        if (c[t].idx >= 0) f(mag_key(c[t].val));
      for (unsigned int t = kK2Cache; t < trips; ++t) {
        const Pair e = entry(t);
        if (e.idx >= 0) f(mag_key(e.val));
      }
    };
    Threshold th;
    if (!band_select_kth(ss, bar, k, pred, ctrl->hist[r], &ctrl->live[r], visit, &th, 250 + 10 * r)) { fail(); return; }
    if (!th.select_all) pred = th.key;  // the prediction for the next union
    trace_stamp(ctrl, 1 + 8 * r + 4);

    // ---- compaction of the winners to where the next phase reads them
    const bool last = r + 1 == rounds;                                  // then me == 0
    const bool send_next = !last && (me & (4u * bit - 1u)) == 2u * bit;  // sender of round r + 1
    const bool only_round = last && copied;
    const bool keep = !last && !send_next;                              // receiver again in round r + 1
    Pair* const OUT = last ? R.gout + (size_t)parity * kcap : R.work[cur_buf ^ 1];
    unsigned long long* const next = R.peer_slots[send_next ? me - 2u * bit : 0u] + slot_off(parity, r + 1, kcap);
    n_cur = th.n < kcap ? th.n : kcap;
    if (cta == 0 && send_next && threadIdx.x == 0) announce(me - 2u * bit, r + 1, n_cur);
    if (cta == 0 && last && threadIdx.x < P && threadIdx.x > 0) announce(threadIdx.x, kFlagBcast, n_cur);
    // keep: the table and (below) the band counts of the next round are built on the way;
    // last: the table over the global set serves the residual put-back, and every peer gets its copy
    auto on_placed = [&](Pair e, unsigned int pos) {
      if (send_next) {
        wire_store(&next[pos], e);
        return;
      }
      if (last)
        for (unsigned int q = 1; q < P; ++q) wire_store(R.peer_slots[q] + slot_off(parity, kFlagBcast, kcap) + pos, e);
      st_pair(&OUT[pos], e);
      if (!only_round) map[e.idx] = (int32_t)pos;
    };
    unsigned int* const tie = &ctrl->tie[r];
    StagedAppender app{&ss, &ctrl->cursor[r], kcap, ctrl, 0u};
    app.begin();
    auto sweep = [&](const Pair (&e)[kK2Cache], unsigned int t0) {
      unsigned int lost = 0;
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        if (t0 + t >= trips) break;
        bool stays = false;
        if (e[t].idx >= 0) {
          stays = passes_threshold(mag_key(e[t].val), th, tie);
          if (stays) {
            app.put(e[t]);
            if (keep) tally(e[t].val, 1u);
          } else {
            lost |= 1u << t;
          }
        }
        app.end_tile(stays, on_placed);
      }
      if (t0 + kK2Cache >= trips) app.flush(on_placed);
      if (!only_round) return;
      // Two ranks: what drops out of A here is not in the global set, and A is this rank's selection.
      float back[kK2Cache];
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        const unsigned int i = (t0 + t) * stride + lane0;
        if (i >= n_a) lost &= ~(1u << t);
        back[t] = 0.f;
        if (lost & (1u << t)) back[t] = R.resid[e[t].idx] + R.sel[i].val;
      }
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t)
        if (lost & (1u << t)) R.resid[e[t].idx] = back[t];
    };
    sweep(c, 0);
    for (unsigned int t0 = kK2Cache; t0 < trips; t0 += kK2Cache) {
      Pair e[kK2Cache];
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) e[t] = entry(t0 + t);
      sweep(e, t0);
    }
    // OUT and map complete; or, when this rank has sent, its work buffers and map free for other use (with two
    // ranks the root has no more use for either)
    if (!only_round && !bar.sync(290 + r)) { fail(); return; }
    trace_stamp(ctrl, 1 + 8 * r + 5);
    if (send_next) {
      trace_stamp(ctrl, 1 + 8 * (r + 1) + 7);
      break;  // left the tree
    }
    if (last) break;
    cur_buf ^= 1;
  }

  // ---- the global set, and the residual put-back of S_local \ S_global
  Pair* const G = R.gout + (size_t)parity * kcap;
  unsigned int n_g = 0;
  if (me == 0u) {  // it has just been written, the table over it too
    n_g = n_cur;
    trace_stamp(ctrl, 40);
    trace_stamp(ctrl, 41);
    if (rounds > 1u) put_back(R.sel, n_sel, G, n_g, map, R.resid, d, cta, nct);
  } else {
    // While the root merges: all of the own selection goes back to the residual, what was there is kept, and
    // the table is built over the selection.  What of it turns out to be in the global set is then undone as
    // its entries come in, with no barrier behind them.  (Table over the global set, barrier, then the put-back:
    // 10 us after the set was there at k = 66 000, 28 us at 255 000.)  One entry at a time: there is time enough, and
    // four in flight take DRAM from the root where ranks share a GPU (k = 255 000: 74.6 -> 77.7 us).
    Pair* const was = R.work[0];
    for (unsigned int i = lane0; i < n_sel; i += stride) {
      Pair e = R.sel[i];
      if ((unsigned int)e.idx < d) {
        map[e.idx] = (int32_t)i;
        const float r0 = R.resid[e.idx];
        R.resid[e.idx] = r0 + e.val;
        e.val = r0;
      }
      st_pair(&was[i], e);
    }
    if (!bar.sync(420)) { fail(); return; }
    if (!cta_wait_flag(sh.ex, R.flags + flag_off(parity, kFlagBcast), epoch, ctrl, limit_ns, 410, &n_g)) {
      fail();
      return;
    }
    if (n_g > kcap) {
      record_error(ctrl, ST_CAPACITY, 411);
      n_g = kcap;
    }
    trace_stamp(ctrl, 40);
    trace_stamp(ctrl, 41);
    unsigned long long* const slot = R.slots + slot_off(parity, kFlagBcast, kcap);
    bool ok = true;
    for (unsigned int i0 = lane0; i0 < n_g && ok; i0 += (unsigned int)kK2Cache * stride) {
      Pair e[kK2Cache];
      unsigned int p[kK2Cache];
      unsigned int want = 0;
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        e[t].idx = -1;
        e[t].val = 0.f;
        if (i0 + t * stride < n_g) want |= 1u << t;
      }
      ok = wire_receive(slot, want, [&](int t) { return (size_t)(i0 + t * stride); }, e, d, ctrl, limit_ns, 412);
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        p[t] = 0xffffffffu;
        if (e[t].idx < 0) continue;
        st_pair(&G[i0 + t * stride], e[t]);
        p[t] = (unsigned int)__ldcg(&map[e[t].idx]);
      }
      Pair w[kK2Cache];
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t) {
        w[t].idx = -1;
        if (p[t] < n_sel) w[t] = ld_pair_cg(&was[p[t]]);
      }
#pragma unroll
      for (int t = 0; t < kK2Cache; ++t)
        if (e[t].idx >= 0 && w[t].idx == e[t].idx) R.resid[e[t].idx] = w[t].val;
    }
    if (!__syncthreads_and(ok)) { fail(); return; }
  }
  trace_stamp(ctrl, 42);
  if (bar.last_arrival()) {  // every CTA is past its last use of the call counter
    if (aborted(ctrl)) {  // a bounds or capacity error that no wait noticed
      fail();
    } else {
      R.n_global[kResCount] = n_g;
      *R.epoch = epoch + 1u;
    }
  }
}

}  // namespace gtk

using namespace gtk;

extern "C" unsigned long long gtk_k2rank_bytes(void) { return sizeof(K2Rank); }

// The small exchange's entries lie behind the flags.
static unsigned long long ll_offset(unsigned long long flags) {
  return (flags + 2ull * kFlagsPerParity * sizeof(uint64_t) + 255ull) & ~255ull;
}

// Symmetric-region geometry, in bytes, for a given kcap: offsets of slots, ag (the wire
// words behind it), gout and flags, and the total size.  out[0..4] = {slots, ag, gout, flags, total}.
extern "C" void gtk_symm_layout(unsigned int kcap, int with_allgather, unsigned long long* out) {
  unsigned long long off = 0;
  out[0] = off;
  off += 2ull * (kMaxRounds + 1) * kcap * sizeof(Pair);
  out[1] = off;
  if (with_allgather) off += 2ull * kMaxPeers * kcap * (sizeof(Pair) + sizeof(unsigned long long));
  out[2] = off;
  off += 2ull * kcap * sizeof(Pair);
  off = (off + 255ull) & ~255ull;
  out[3] = off;
  off = ll_offset(off);
  off += 2ull * (kMaxRounds + 1) * kLLMaxK * sizeof(ulonglong2);
  out[4] = off;
}

// Fill one K2Rank descriptor on the host (the caller copies it to the device).
extern "C" int gtk_k2rank_fill(void* desc_host, const void* sel, unsigned int sel_cap, const void* st, void* work0,
                               void* work1, void* map, void* resid, void* symm_local, void* ctrl,
                               void* n_global, void* epoch_word, unsigned int kcap,
                               int with_allgather, unsigned int P, void* const* symm_peers) {
  if (P > (unsigned int)kMaxPeers) return GTK_ERR_ARG;
  unsigned long long lay[5];
  gtk_symm_layout(kcap, with_allgather, lay);
  K2Rank* r = (K2Rank*)desc_host;
  r->sel = (const Pair*)sel;
  r->sel_cap = sel_cap;
  r->st = (const K1State*)st;
  r->work[0] = (Pair*)work0;
  r->work[1] = (Pair*)work1;
  r->map = (int32_t*)map;
  r->resid = (float*)resid;
  char* base = (char*)symm_local;
  r->slots = (unsigned long long*)(base + lay[0]);
  r->ag = (Pair*)(base + lay[1]);
  const unsigned long long wire = lay[1] + 2ull * kMaxPeers * kcap * sizeof(Pair);
  r->wire = (unsigned long long*)(base + wire);
  r->gout = (Pair*)(base + lay[2]);
  r->flags = (uint64_t*)(base + lay[3]);
  r->ll = (ulonglong2*)(base + ll_offset(lay[3]));
  r->ctrl = (Ctrl*)ctrl;
  r->n_global = (unsigned int*)n_global;
  r->epoch = (unsigned int*)epoch_word;
  for (unsigned int q = 0; q < (unsigned int)kMaxPeers; ++q) {
    char* pb = q < P ? (char*)symm_peers[q] : nullptr;
    r->peer_slots[q] = pb ? (unsigned long long*)(pb + lay[0]) : nullptr;
    r->peer_ag[q] = pb ? (Pair*)(pb + lay[1]) : nullptr;
    r->peer_wire[q] = pb ? (unsigned long long*)(pb + wire) : nullptr;
    r->peer_flags[q] = pb ? (uint64_t*)(pb + lay[3]) : nullptr;
    r->peer_ll[q] = pb ? (ulonglong2*)(pb + ll_offset(lay[3])) : nullptr;
  }
  return GTK_OK;
}

static int k2_max_coresident() {
  static int cached = 0;  // the occupancy query costs microseconds; the answer never changes
  if (cached) return cached;
  const DeviceInfo* di = gtk_device_info();
  if (!di) return 0;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)k2_gtopk_exchange, kSelThreads, 0) !=
      cudaSuccess)
    return 0;
  cached = occ * di->sms;
  return cached;
}

// Largest cluster (CTAs of one rank joined by the hardware barrier) that `nranks` ranks can hold
// co-resident on this device; 0 if clusters cannot be used.  Cached per (nranks, nctas).
static bool k2_cluster_fits(unsigned int nranks, unsigned int nctas) {
  static int cache[kMaxPeers + 1][17] = {};  // 0 unknown, 1 yes, 2 no
  if (nctas < 2 || nctas > 16 || (nctas & (nctas - 1)) || nranks > (unsigned int)kMaxPeers) return false;
  int& c = cache[nranks][nctas];
  if (c) return c == 1;
  c = 2;
  const DeviceInfo* di = gtk_device_info();
  if (!di || !di->cluster) return false;
  if (nctas > 8 && cudaFuncSetAttribute((const void*)k2_gtopk_exchange,
                                        cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nctas, nranks);
  cfg.blockDim = dim3(kSelThreads);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nclusters = 0;
  if (cudaOccupancyMaxActiveClusters(&nclusters, (const void*)k2_gtopk_exchange, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (nclusters < (int)nranks) return false;
  c = 1;
  return true;
}

// ranks_dev: device array of nranks_in_launch K2Rank descriptors (1 in production).  Nothing is
// cleared here: the kernel alternates between the two control blocks of each rank.
// use_cluster: 1 = join the CTAs of a rank into one thread-block cluster (hardware barrier) when
// nctas is 2, 4, 8 or 16 and the device can hold the clusters; 0 = software barrier.
extern "C" int gtk_k2_exchange(const void* ranks_dev, unsigned int nranks, unsigned int rank_base,
                               unsigned int P, unsigned int k, unsigned int kcap, unsigned int d,
                               unsigned int nctas, unsigned long long limit_ns, int use_cluster,
                               void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (P < 2 || (P & (P - 1)) != 0 || P > (unsigned int)kMaxPeers) return GTK_ERR_ARG;
  if (k == 0 || k > kcap || nranks == 0 || nctas == 0) return GTK_ERR_ARG;
  const K2Rank* ranks = (const K2Rank*)ranks_dev;
  if (k2_small_serves(nranks, k, nctas))
    return k2_small_launch(ranks, nranks, rank_base, P, k, kcap, d, limit_ns, stream);
  int cluster = (use_cluster && k2_cluster_fits(nranks, nctas)) ? 1 : 0;
  const auto fn = k2_gtopk_exchange;
  if ((int)(nranks * nctas) > k2_max_coresident()) return GTK_ERR_ARG;
  void* args[] = {&ranks, &rank_base, &P, &k, &kcap, &d, &limit_ns, &cluster};
  cudaError_t e;
  if (cluster) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nctas, nranks);
    cfg.blockDim = dim3(kSelThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;  // several emulated ranks wait on one another
    attr[1].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = nranks > 1 ? 2 : 1;  // one cluster is co-scheduled by the hardware anyway
    e = cudaLaunchKernelExC(&cfg, (const void*)fn, args);
  } else if (nranks * nctas == 1) {
    // one CTA waits on nobody of its own launch: a plain launch
    fn<<<dim3(1, 1), dim3(kSelThreads), 0, stream>>>(ranks, rank_base, P, k, kcap, d, limit_ns, 0);
    e = cudaGetLastError();
  } else {
    e = cudaLaunchCooperativeKernel((void*)fn, dim3(nctas, nranks), dim3(kSelThreads), args, 0, stream);
  }
  gtk_count_launch(1);
  if (e != cudaSuccess) return GTK_ERR_CUDA;
  return GTK_OK;
}
