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
#include "exchange_common.cuh"

namespace gtk {

__global__ void __launch_bounds__(kSelThreads)
k2t_topk_allgather(const K2Rank* __restrict__ ranks, unsigned int rank_base, unsigned int P,
                   unsigned int k, unsigned int kcap, unsigned int work_cap, unsigned int d,
                   int reselect, unsigned int* __restrict__ seg_counts_all,
                   unsigned long long limit_ns) {
  __shared__ ExchangeShared sh;
  __shared__ unsigned int band[kHistBins];  // this CTA's share of the first selection level, counted on the fly
  __shared__ unsigned int counts[kMaxPeers];
  const K2Rank& R = ranks[blockIdx.y];
  const unsigned int epoch = __ldcg(R.epoch);
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
  if (__ldcg(&R.n_global[kResStatus]) != 0u) {
    if (cta == 0 && threadIdx.x < (unsigned int)kMaxPeers) seg_counts[threadIdx.x] = 0u;
    if (cta == 0 && threadIdx.x == 0) R.n_global[kResCount] = 0u;
    return;
  }

  unsigned int n_sel = R.st->n_sel;
  if (n_sel > kcap) n_sel = kcap;

  // push my selection into slot[me] of every rank (my own included)
  for (unsigned int q = 0; q < P; ++q) {
    Pair* dst = (q == me ? R.ag : R.peer_ag[q]) + ag_off(parity, me, kcap);
    push_pairs(dst, R.sel, n_sel, cta, nct);
  }
  cta_fence_peer_stores(nct == 1);
  if (!bar.sync(500)) { fail(); return; }
  if (cta == 0 && threadIdx.x < P && threadIdx.x != me)  // one releasing thread per destination
    release_flag(R.peer_flags[threadIdx.x] + flag_off(parity, kFlagAg0 + me), epoch, n_sel);
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
  const uint32_t pred = mag_key(R.st->kth_mag);  // no sum of P selections has its k-th magnitude below the own one
  for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) band[i] = 0u;
  __syncthreads();
  auto tally = [&](float v, unsigned int delta) { atomicAdd(&band[band_bin(mag_key(v), pred)], delta); };
  Pair* A = R.work[0];
  const Pair* L0 = R.ag + ag_off(parity, 0, kcap);
  copy_and_map(A, L0, counts[0], R.map, d, cta, nct, ctrl, tally);
  unsigned int n_a = counts[0];
  if (cta == 0 && threadIdx.x == 0) ctrl->n_live = n_a;
  if (!bar.sync(540)) { fail(); return; }
  const unsigned int stride = nct * kSelThreads;
  for (unsigned int q = 1; q < P; ++q) {
    const Pair* B = R.ag + ag_off(parity, q, kcap);
    const unsigned int n_b = counts[q];
    const unsigned int trips = (n_b + stride - 1) / stride;
    for (unsigned int t = 0; t < trips; ++t) {
      const unsigned int j = t * stride + cta * kSelThreads + threadIdx.x;
      bool append = false;
      Pair e;
      e.idx = -1;
      e.val = 0.f;
      if (j < n_b) {
        e = ld_pair_cg(&B[j]);
        if ((unsigned int)e.idx >= d) {
          record_error(ctrl, ST_BOUNDS, 550);
        } else {
          append = true;
          const unsigned int p = (unsigned int)__ldcg(&R.map[e.idx]);
          if (p < n_a) {
            const Pair a = ld_pair_cg(&A[p]);
            if (a.idx == e.idx) {
              const float sum = a.val + e.val;
              A[p].val = sum;
              tally(a.val, 0xffffffffu);
              tally(sum, 1u);
              append = false;
            }
          }
        }
      }
      const unsigned int m = __ballot_sync(0xffffffffu, append);
      if (m) {
        unsigned int base = 0;
        if (lane_id() == (unsigned int)(__ffs(m) - 1)) base = atomicAdd(&ctrl->n_live, __popc(m));
        base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
        if (append) {
          const unsigned int pos = base + __popc(m & lanemask_lt());
          if (pos < work_cap) {
            st_pair(&A[pos], e);
            R.map[e.idx] = (int32_t)pos;
            tally(e.val, 1u);
          } else {
            record_error(ctrl, ST_CAPACITY, 551);
          }
        }
      }
    }
    if (q + 1u == P) {  // the sums are final: publish this CTA's counts
      __syncthreads();
      for (int i = threadIdx.x; i < kHistBins; i += kSelThreads) {
        const unsigned int n = band[i];
        if (n) atomicAdd(&ctrl->hist[0][0][i], n);
      }
    }
    if (!bar.sync(560 + q)) { fail(); return; }
    n_a = __ldcg(&ctrl->n_live);
    if (n_a > work_cap) n_a = work_cap;
  }
  auto visit = [&](auto f) {
    for (unsigned int i = cta * kSelThreads + threadIdx.x; i < n_a; i += stride) f(mag_key(ld_pair_cg(&A[i]).val));
  };
  Threshold th;
  if (!band_select_kth(sh.sel, bar, k, pred, ctrl->hist[0], &ctrl->live[0], visit, &th, 580)) { fail(); return; }
  Pair* G = R.gout + (size_t)parity * kcap;
  int32_t* map = R.map;
  auto on_placed = [&](Pair e, unsigned int pos) {
    st_pair(&G[pos], e);
    map[e.idx] = (int32_t)pos;
  };
  StagedAppender app{&sh.sel, &ctrl->cursor[0], kcap, ctrl};
  app.begin();
  const unsigned int trips = (n_a + stride - 1) / stride;
  for (unsigned int t = 0; t < trips; ++t) {
    const unsigned int i = t * stride + cta * kSelThreads + threadIdx.x;
    if (i < n_a) {
      const Pair e = ld_pair_cg(&A[i]);
      if (passes_threshold(mag_key(e.val), th, &ctrl->tie[0])) app.put(e);
    }
    app.end_tile(on_placed);
  }
  app.flush(on_placed);
  if (!bar.sync(590)) { fail(); return; }
  unsigned int n_g = __ldcg(&ctrl->cursor[0]);
  if (n_g > kcap) n_g = kcap;
  put_back(R.sel, n_sel, G, n_g, R.map, R.resid, d, cta, nct);
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
