// K2t: Top-k all-gather exchange ('topk') and its re-selecting variant ('topk2').
//
// 'topk'  (allreducer.py:29-64 + 461-466 in the reference): every rank ends
//         with all P selections; the dense result is the sum of the P sparse
//         vectors, nothing returns to the residual.  Here each rank pushes its k
//         pairs into slot[rank] of every peer with NVLink peer stores and one
//         flag per source; the consumer (K3, atomic mode) applies the P segments.
// 'topk2' (allreducer.py:467-473): the summed vector is re-sparsified to its k
//         largest magnitudes, and locally selected entries that did not survive
//         return to the residual.  Here the P lists are merged in rank order
//         (same arithmetic on every rank, so all ranks get the same set) with
//         the direct-address table, then radix-selected.
//
// What bounds topk2: a barrier per merged list and three round trips between
// them (table, entry, append).  The lists travel as the tree's 8-byte wire words,
// so nobody fences or waits for a complete list, and a merged entry remembers
// where in the own selection it comes from, so that dropping it is also its way
// back to the residual.  Four ranks, k = 14 728, the same selection again and again:
// 53 us with flags behind fenced stores, the put-back behind a table over the global
// set and one entry per thread in flight, 29 now (eight ranks, k = 20 000: 139 and
// 76; two, k = 660 340: 312 and 176; 'topk', four ranks, k = 14 728: 23 and 10).
#include "exchange_common.cuh"

namespace gtk {

constexpr int kBatch = 4;                         // entries per thread whose loads are in flight together
constexpr unsigned int kNotOwn = 0xffffffffu;

__global__ void __launch_bounds__(kSelThreads, 2)
k2t_topk_allgather(const K2Rank* __restrict__ ranks, unsigned int rank_base, unsigned int P,
                   unsigned int k, unsigned int kcap, unsigned int work_cap, unsigned int d,
                   int reselect, unsigned int* __restrict__ seg_counts_all,
                   unsigned long long limit_ns) {
  __shared__ ExchangeShared sh;
  __shared__ unsigned int band[kHistBins];  // this CTA's share of the first selection level, counted on the fly
  __shared__ unsigned int counts[kMaxPeers];
  const K2Rank& R = ranks[blockIdx.y];
  // One round of loads (a load behind the check of the status would be another round trip).
  const unsigned int epoch = __ldcg(R.epoch);
  const unsigned int status = __ldcg(&R.n_global[kResStatus]);
  unsigned int n_sel = __ldcg(&R.st->n_sel);
  const float kth_mag = __ldcg(&R.st->kth_mag);
  const unsigned int me = rank_base + blockIdx.y;
  const unsigned int cta = blockIdx.x, nct = gridDim.x;
  const unsigned int parity = epoch & 1u;
  Ctrl* ctrl = R.ctrl + parity;
  RankBarrier bar{ctrl, nct, 0u, limit_ns};
  unsigned int* seg_counts = seg_counts_all + (size_t)blockIdx.y * kMaxPeers;

  // A call that gives up leaves EMPTY results (no segment, no global pair: the consumer applies
  // nothing) and a sticky status; later calls return at once until the host rebuilds the exchange.
  auto fail = [&]() {
    if (threadIdx.x == 0) {
      atomicExch(&R.n_global[kResCount], 0u);
      for (unsigned int q = 0; q < (unsigned int)kMaxPeers; ++q) seg_counts[q] = 0u;
      unsigned int st = ld_relaxed_gpu_u32(&ctrl->status);
      if (st == 0u) st = ST_TIMEOUT_BARRIER;
      if (atomicCAS(&R.n_global[kResStatus], 0u, st) == 0u) {
        R.n_global[kResWhere] = ld_relaxed_gpu_u32(&ctrl->where);
        R.n_global[kResEpoch] = epoch;
      }
    }
  };
  if (status != 0u) {
    if (cta == 0 && threadIdx.x < (unsigned int)kMaxPeers) seg_counts[threadIdx.x] = 0u;
    if (cta == 0 && threadIdx.x == 0) R.n_global[kResCount] = 0u;
    return;
  }

  if (n_sel > kcap) n_sel = kcap;

  const unsigned int stride = nct * kSelThreads;
  const unsigned int lane0 = cta * kSelThreads + threadIdx.x;

  // push my selection into slot[me] of every rank (topk: my own included)
  if (reselect) {  // words that say themselves that they have arrived, in no order with the counts
    if (cta == 0 && threadIdx.x < P && threadIdx.x != me)
      st_relaxed_sys_u64(reinterpret_cast<unsigned long long*>(R.peer_flags[threadIdx.x] + flag_off(parity, kFlagAg0 + me)),
                         ((unsigned long long)epoch << 32) | n_sel);
    for_pairs(R.sel, n_sel, lane0, stride, [&](Pair e, unsigned int i) {
      for (unsigned int q = 0; q < P; ++q)
        if (q != me) wire_store(R.peer_wire[q] + ag_off(parity, me, kcap) + i, e);
    });
  } else {
    for_pairs(R.sel, n_sel, lane0, stride, [&](Pair e, unsigned int i) {
      for (unsigned int q = 0; q < P; ++q) st_pair(R.peer_ag[q] + ag_off(parity, me, kcap) + i, e);
    });
    cta_fence_peer_stores(nct == 1);
    if (!bar.sync(500)) { fail(); return; }
    if (cta == 0 && threadIdx.x < P && threadIdx.x != me)  // one releasing thread per destination
      release_flag(R.peer_flags[threadIdx.x] + flag_off(parity, kFlagAg0 + me), epoch, n_sel);
  }
  // wait for every source, one polling thread for each
  if (threadIdx.x == 0) sh.ok = 1;
  __syncthreads();
  if (threadIdx.x < P) {
    const unsigned int q = threadIdx.x;
    unsigned int c = n_sel;
    if (q != me && !wait_flag(R.flags + flag_off(parity, kFlagAg0 + q), epoch, ctrl, limit_ns, 510 + q, &c)) {
      sh.ok = 0;
      c = 0u;
    }
    if (c > kcap) {
      record_error(ctrl, ST_CAPACITY, 530 + q);
      c = kcap;
    }
    counts[q] = c;
  }
  __syncthreads();
  if (!sh.ok) { fail(); return; }
  // The other control block, for the next call (what this form dirties of it: header, stamps, one histogram set).
  {
    uint4* other = reinterpret_cast<uint4*>(R.ctrl + (parity ^ 1u));
    const size_t nvec16 = (offsetof(Ctrl, hist) + sizeof(((Ctrl*)0)->hist[0])) / 16;
    for (size_t i = cta * kSelThreads + threadIdx.x; i < nvec16; i += (size_t)nct * kSelThreads)
      other[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (!reselect) {
    if (bar.last_arrival()) {  // every CTA has read the epoch word
      if (aborted(ctrl)) {
        fail();
      } else {
        for (unsigned int q = 0; q < P; ++q) seg_counts[q] = counts[q];
        *R.epoch = epoch + 1u;
      }
    }
    return;
  }

  // ---- topk2: merge the P lists in rank order, then keep the k largest sums
  // A prediction, as in the tree: the sums' k-th magnitude lies below the own one where entries cancel.
  const uint32_t pred = mag_key(kth_mag);
  for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) band[i] = 0u;
  __syncthreads();
  auto tally = [&](float v, unsigned int delta) { atomicAdd(&band[band_bin(mag_key(v), pred)], delta); };
  Pair* const A = R.work[0];
  int32_t* const map = R.map;
  unsigned int* const own = reinterpret_cast<unsigned int*>(R.work[1]);  // A's entry i: where in the own selection, or kNotOwn
  Pair c[kBatch];
  // Takes trips t0 .. t0 + kBatch - 1 of list q into c[] (idx -1: none); slot q keeps them as in topk.
  auto fetch = [&](unsigned int q, unsigned int t0) {
    const unsigned int n = counts[q];
    unsigned int want = 0;
    bool ok = true;
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {
      const unsigned int j = (t0 + t) * stride + lane0;
      c[t].idx = -1;
      c[t].val = 0.f;
      if (j < n) want |= 1u << t;
    }
    if (q != me) {
      ok = wire_receive(R.wire + ag_off(parity, q, kcap), want,
                        [&](int t) { return (size_t)((t0 + t) * stride + lane0); }, c, d, ctrl, limit_ns, 510 + q);
    } else {
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        if (!(want & (1u << t))) continue;
        c[t] = ld_pair_cg(&R.sel[(t0 + t) * stride + lane0]);
        if ((unsigned int)c[t].idx >= d) {
          record_error(ctrl, ST_BOUNDS, 550);
          c[t].idx = -1;
        }
      }
    }
    Pair* const slot = R.ag + ag_off(parity, q, kcap);
#pragma unroll
    for (int t = 0; t < kBatch; ++t)
      if (want & (1u << t)) st_pair(&slot[(t0 + t) * stride + lane0], c[t]);
    return ok;
  };
  // Entries that list q adds are counted in scratch[q mod 3]: the union's size before the list must not move
  // while slower CTAs read it, or a look-up could take an entry of an earlier call for one of this.  The word of
  // list q + 1 was last read before the barrier behind list q - 1.
  unsigned int n_a = 0;
  for (unsigned int q = 0; q < P; ++q) {
    unsigned int* const added = &ctrl->scratch[q % 3u];
    const unsigned int trips = (counts[q] + stride - 1) / stride;
    // a list's first entries come in while the one before is being completed
    if (!__syncthreads_and(fetch(q, 0))) { fail(); return; }
    if (q != 0u) {
#pragma unroll
      for (int t = 0; t < kBatch; ++t) prefetch_entry(map, c[t].idx, d);
      if (!bar.wait(560 + q)) { fail(); return; }
      n_a = q == 1u ? counts[0] : n_a + __ldcg(&ctrl->scratch[(q - 1u) % 3u]);
      if (n_a > work_cap) n_a = work_cap;
    }
    if (cta == 0 && threadIdx.x == 0) ctrl->scratch[(q + 1u) % 3u] = 0u;
    for (unsigned int t0 = 0; t0 < trips; t0 += kBatch) {
      if (t0 != 0u && !__syncthreads_and(fetch(q, t0))) { fail(); return; }
      unsigned int pm[kBatch], fresh[kBatch];
      Pair a[kBatch];
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        pm[t] = 0xffffffffu;
        if (q != 0u && c[t].idx >= 0) pm[t] = (unsigned int)__ldcg(&map[c[t].idx]);
      }
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        a[t].idx = -1;
        a[t].val = 0.f;
        if (pm[t] < n_a) a[t] = ld_pair_cg(&A[pm[t]]);
      }
      unsigned int n_fresh = 0;  // of this warp
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        const bool shared = c[t].idx >= 0 && a[t].idx == c[t].idx;
        if (shared) {
          const float sum = a[t].val + c[t].val;
          A[pm[t]].val = sum;
          if (q == me) own[pm[t]] = (t0 + t) * stride + lane0;
          tally(a[t].val, 0xffffffffu);
          tally(sum, 1u);
          c[t].idx = -1;
        }
        fresh[t] = __ballot_sync(0xffffffffu, c[t].idx >= 0);
        n_fresh += __popc(fresh[t]);
      }
      unsigned int base = 0;
      if (q != 0u && n_fresh && lane_id() == 0) base = n_a + atomicAdd(added, n_fresh);
      base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        if (c[t].idx >= 0) {
          // (the first list keeps its order: no counter, no round trip)
          const unsigned int pos = q == 0u ? (t0 + t) * stride + lane0 : base + __popc(fresh[t] & lanemask_lt());
          if (pos < work_cap) {
            st_pair(&A[pos], c[t]);
            own[pos] = q == me ? (t0 + t) * stride + lane0 : kNotOwn;
            map[c[t].idx] = (int32_t)pos;
            tally(c[t].val, 1u);
          } else {
            record_error(ctrl, ST_CAPACITY, 551);
          }
        }
        base += __popc(fresh[t]);
      }
    }
    if (q + 1u == P) {  // the sums are final: publish this CTA's counts
      __syncthreads();
      for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) {
        const unsigned int n = band[i];
        if (n) atomicAdd(&ctrl->hist[0][0][i], n);
      }
    }
    bar.arrive();
  }
  if (!bar.wait(560 + P)) { fail(); return; }
  n_a += __ldcg(&ctrl->scratch[(P - 1u) % 3u]);  // (two ranks at least)
  if (n_a > work_cap) n_a = work_cap;
  const unsigned int trips = (n_a + stride - 1) / stride;
  auto load = [&](Pair (&e)[kBatch], unsigned int t0) {
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {
      const unsigned int i = (t0 + t) * stride + lane0;
      e[t].idx = -1;
      e[t].val = 0.f;
      if (i < n_a) e[t] = ld_pair_cg(&A[i]);
    }
  };
  load(c, 0);  // kept in registers for both sweeps
  auto visit = [&](auto f) {
#pragma unroll
    for (int t = 0; t < kBatch; ++t)
      if (c[t].idx >= 0) f(mag_key(c[t].val));
    for (unsigned int t0 = kBatch; t0 < trips; t0 += kBatch) {
      Pair e[kBatch];
      load(e, t0);
#pragma unroll
      for (int t = 0; t < kBatch; ++t)
        if (e[t].idx >= 0) f(mag_key(e[t].val));
    }
  };
  Threshold th;
  if (!band_select_kth(sh.sel, bar, k, pred, ctrl->hist[0], &ctrl->live[0], visit, &th, 580)) { fail(); return; }
  Pair* const G = R.gout + (size_t)parity * kcap;
  auto on_placed = [&](Pair e, unsigned int pos) { st_pair(&G[pos], e); };
  StagedAppender app{&sh.sel, &ctrl->cursor[0], kcap, ctrl, 0u};
  app.begin();
  auto sweep = [&](const Pair (&e)[kBatch], unsigned int t0) {
    unsigned int from[kBatch];
    float back[kBatch];
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {
      from[t] = kNotOwn;
      bool stays = false;
      if (e[t].idx >= 0) {
        stays = passes_threshold(mag_key(e[t].val), th, &ctrl->tie[0]);
        if (stays) app.put(e[t]);
        else from[t] = __ldcg(&own[(t0 + t) * stride + lane0]);
      }
      if (t0 + t < trips) app.end_tile(stays, on_placed);
    }
    // what drops out of the sum although this rank had selected it goes back to its residual
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {
      back[t] = 0.f;
      if (from[t] != kNotOwn) back[t] = R.resid[e[t].idx] + R.sel[from[t]].val;
    }
#pragma unroll
    for (int t = 0; t < kBatch; ++t)
      if (from[t] != kNotOwn) R.resid[e[t].idx] = back[t];
  };
  sweep(c, 0);
  for (unsigned int t0 = kBatch; t0 < trips; t0 += kBatch) {
    Pair e[kBatch];
    load(e, t0);
    sweep(e, t0);
  }
  app.flush(on_placed);
  const unsigned int n_g = th.n < kcap ? th.n : kcap;
  if (bar.last_arrival()) {
    if (aborted(ctrl)) {
      fail();
    } else {
      for (unsigned int q = 0; q < P; ++q) seg_counts[q] = counts[q];
      R.n_global[kResCount] = n_g;
      *R.epoch = epoch + 1u;
    }
  }
}

}  // namespace gtk

using namespace gtk;

// Nothing is cleared here: the kernel alternates between the two control blocks of each rank.
extern "C" int gtk_k2t_allgather(const void* ranks_dev, unsigned int nranks, unsigned int rank_base, unsigned int P,
                                 unsigned int k, unsigned int kcap, unsigned int work_cap, unsigned int d,
                                 int reselect, void* seg_counts,
                                 unsigned int nctas, unsigned long long limit_ns, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (P < 2 || P > (unsigned int)kMaxPeers) return GTK_ERR_ARG;
  if (k == 0 || k > kcap || nranks == 0 || nctas == 0) return GTK_ERR_ARG;
  const DeviceInfo* di = gtk_device_info();
  if (!di) return GTK_ERR_CUDA;
  static int occ = 0;
  if (!occ && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)k2t_topk_allgather,
                                                            kSelThreads, 0) != cudaSuccess)
    return GTK_ERR_CUDA;
  if ((int)(nranks * nctas) > occ * di->sms) return GTK_ERR_ARG;
  const K2Rank* ranks = (const K2Rank*)ranks_dev;
  unsigned int* segc = (unsigned int*)seg_counts;
  void* args[] = {&ranks, &rank_base, &P, &k, &kcap, &work_cap, &d, &reselect, &segc, &limit_ns};
  cudaError_t e = cudaLaunchCooperativeKernel((void*)k2t_topk_allgather, dim3(nctas, nranks),
                                              dim3(kSelThreads), args, 0, stream);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}
