// K3: sparse scatter + averaging + weight decay + momentum/nesterov SGD over the
// flat parameter and momentum buffers.
//
// Replaces, in the reference: fill_(0) + scatter of the global values + "/= P"
// (allreducer.py:458-475) and the per-parameter SGD loop of
// distributed_optimizer.py:105-143 (d_p += wd*p; buf = m*buf + d_p, first step
// buf = d_p; nesterov d_p += m*buf; p -= lr*d_p), three launches per tensor.
//
// The update is split so that the dense gradient is never built:
//   dense part   g = wd*p (+ coef*scale*g_dense in dense mode);
//                buf = m*buf + f*g;  p -= lr*(nesterov ? g + m*buf : buf)
//                -- independent of the exchange, so it may run while K2 is in flight.
//   sparse part  for each global pair (j, v): s = coef*scale*v, sb = f*s;
//                buf[j] += sb;  p[j] -= lr*(nesterov ? s + m*sb : sb)
// where f = 1 on the first step and 1 - dampening afterwards.  Both parts add up
// to the reference's update because it is affine in the gradient.
#include "exchange_common.cuh"
#include "launch.cuh"
#include "host_api.h"

namespace gtk {

constexpr int kK3Threads = 512;

// Sparse inputs may live in a two-parity buffer written by the exchange kernel:
// the segment base is pairs + ((*parity_word - 1) & 1) * parity_stride, where
// parity_word is the exchange's call counter after the call (nullptr: no offset).
__device__ __forceinline__ const Pair* parity_base(const Pair* pairs, const unsigned int* parity_word,
                                                   unsigned int parity_stride) {
  if (!parity_word) return pairs;
  return pairs + (size_t)((*parity_word - 1u) & 1u) * parity_stride;
}

struct SgdHyper {
  const float* lr_ptr;  // device-resident learning rate (read when non-null; lets a captured graph follow a schedule)
  float lr;
  float momentum;
  float dampening;
  float weight_decay;
  int nesterov;
  int first_step;
};

template <bool HAS_G, bool HAS_BUF>
__global__ void __launch_bounds__(kK3Threads, 2)
k3_dense(float* p, float* buf, const float* g,
         const float* coef_ptr, float scale, long long d, SgdHyper h) {
  pdl_begin(p, buf, g, coef_ptr, h.lr_ptr);
  if (h.lr_ptr) h.lr = *h.lr_ptr;
  const float coef = (HAS_G && coef_ptr) ? (*coef_ptr) * scale : scale;
  const float f = h.first_step ? 1.0f : 1.0f - h.dampening;
  const float m = h.momentum;
  auto upd = [&](float& pj, float& bj, float gj) {
    float gr = h.weight_decay * pj;
    if (HAS_G) gr = fmaf(gj, coef, gr);
    float step = gr;
    if (HAS_BUF) {
      bj = fmaf(m, bj, f * gr);
      step = h.nesterov ? fmaf(m, bj, gr) : bj;
    }
    pj = fmaf(-h.lr, step, pj);
  };
  const unsigned int mis = (unsigned int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3u);
  long long head = mis ? (4 - mis) : 0;
  if (head > d) head = d;
  const long long nvec = (d - head) >> 2;
  const long long tail0 = head + (nvec << 2);
  float4* p4 = reinterpret_cast<float4*>(p + head);
  float4* b4 = reinterpret_cast<float4*>(buf + head);
  const float4* g4 = reinterpret_cast<const float4*>(g + head);
  const long long stride = (long long)gridDim.x * kK3Threads;
  for (long long v = (long long)blockIdx.x * kK3Threads + threadIdx.x; v < nvec; v += 2 * stride) {
    const long long v1 = v + stride;
    const bool two = v1 < nvec;
    float4 pa = p4[v], pb = two ? p4[v1] : make_float4(0, 0, 0, 0);
    float4 ba = make_float4(0, 0, 0, 0), bb = ba, ga = ba, gb = ba;
    if (HAS_BUF) { ba = b4[v]; if (two) bb = b4[v1]; }
    if (HAS_G) { ga = __ldcs(&g4[v]); if (two) gb = __ldcs(&g4[v1]); }
    upd(pa.x, ba.x, ga.x); upd(pa.y, ba.y, ga.y); upd(pa.z, ba.z, ga.z); upd(pa.w, ba.w, ga.w);
    p4[v] = pa;
    if (HAS_BUF) b4[v] = ba;
    if (two) {
      upd(pb.x, bb.x, gb.x); upd(pb.y, bb.y, gb.y); upd(pb.z, bb.z, gb.z); upd(pb.w, bb.w, gb.w);
      p4[v1] = pb;
      if (HAS_BUF) b4[v1] = bb;
    }
  }
  if (blockIdx.x == 0) {
    const long long nscalar = head + (d - tail0);
    for (long long j = threadIdx.x; j < nscalar; j += kK3Threads) {
      const long long i = j < head ? j : tail0 + (j - head);
      float pj = p[i], bj = HAS_BUF ? buf[i] : 0.f, gj = HAS_G ? g[i] : 0.f;
      upd(pj, bj, gj);
      p[i] = pj;
      if (HAS_BUF) buf[i] = bj;
    }
  }
}

// Sparse part.  `pairs` holds nseg segments of seg_stride pairs; segment s (one row of the grid) has
// counts[s] live pairs.  use_atomics: indices may repeat across segments.
// What bounds it: scattered 4-byte accesses, each a 32-byte sector of DRAM read and written back (about 23 pairs a ns).
// One entry per thread and as many CTAs as that takes: CTAs that have loaded and CTAs that store are then always
// there side by side.  With four entries per thread in a grid that fills the chip once, all of it loads first and
// stores afterwards: select + update of 138 M elements at 0.01 353 us against 337, with momentum 422 against 397
// (60 M: 191 and 181; two entries per thread: 340, 408 and 188); the same up to 300 000 entries.
// The lists may be far shorter than their buffers (four times after the first epoch of the default schedule), and then
// reading up to the buffers' end, or CTAs without entries, are most of what there is to do.  So the grid goes by the
// caller's count where there is one, it ends at four times what the chip holds (1.2 M entries over all lists; the threads
// loop from there on), and entries are read ahead of the counts only where they are few.  Against a grid and a read-ahead
// up to the buffers' size, without a count and with it: eight lists of 138 000 entries in four times the room 55.0, 43.5
// and 43.5 us, eight of 13 800 in 40 times 22.7, 10.3 and 9.5, one of 345 000 in four times 9.5, 8.5 and 7.5; a full
// one of 1.38 M 63.0 and 63.5, where two times what the chip holds takes 65.2.
constexpr int kSparseThreads = 256;
constexpr unsigned int kSparseMaxBlocks = 4u * 148u * 8u;  // (148 SMs with 2 048 threads each)
constexpr unsigned long long kSparseAhead = 1ull << 18;  // entries over all lists
__global__ void __launch_bounds__(kSparseThreads)
k3_sparse(float* p, float* buf, const Pair* pairs,
          const unsigned int* counts, unsigned int seg_stride,
          const float* coef_ptr, float scale, unsigned int d, SgdHyper h,
          int use_atomics, unsigned int* bad_index_count,
          const unsigned int* parity_word, unsigned int parity_stride, int ahead) {
  pdl_begin(p, buf, pairs, counts, coef_ptr, parity_word, h.lr_ptr);
  const Pair* seg = pairs + (size_t)blockIdx.y * seg_stride;
  const unsigned int stride = gridDim.x * kSparseThreads;
  unsigned int i = blockIdx.x * kSparseThreads + threadIdx.x;
  // One round of loads.  ahead: the lists are there up to their capacity, so that a thread reads its first entry
  // (of both halves) before it knows how many are valid.  (Read behind the counts: select + update of 3 M elements at
  // 0.003 17.5 us against 17.25, 8 M at 0.002 31.2 and 31.0, all-gather of 4 x 16 000 and update 13.0 and 12.4.)
  Pair e[2];
  e[0].idx = e[1].idx = 0;
  e[0].val = e[1].val = 0.f;
  if (ahead && i < seg_stride) {
    e[0] = seg[i];
    if (parity_word) e[1] = seg[parity_stride + i];
  }
  unsigned int n = counts[blockIdx.y];
  const unsigned int half = parity_word ? (*parity_word - 1u) & 1u : 0u;
  if (h.lr_ptr) h.lr = *h.lr_ptr;
  const float coef = coef_ptr ? (*coef_ptr) * scale : scale;
  const float f = h.first_step ? 1.0f : 1.0f - h.dampening;
  const bool has_buf = buf != nullptr && h.momentum != 0.f;
  if (n > seg_stride) n = seg_stride;
  seg += (size_t)half * parity_stride;
  auto apply = [&](Pair x) {
    if ((unsigned int)x.idx >= d) {
      atomicAdd(bad_index_count, 1u);
      return;
    }
    float pv = 0.f, bv = 0.f;
    if (!use_atomics) {
      pv = p[x.idx];
      if (has_buf) bv = buf[x.idx];
    }
    const float sv = x.val * coef;
    float step = sv;
    if (has_buf) {
      const float sb = f * sv;
      if (use_atomics) atomicAdd(&buf[x.idx], sb);
      else buf[x.idx] = bv + sb;
      step = h.nesterov ? fmaf(h.momentum, sb, sv) : sb;
    }
    if (use_atomics) atomicAdd(&p[x.idx], -h.lr * step);
    else p[x.idx] = fmaf(-h.lr, step, pv);
  };
  if (ahead && i < n) {
    apply(half ? e[1] : e[0]);
    i += stride;
  }
  for (; i < n; i += stride) apply(seg[i]);
}

// Optional: build the dense averaged gradient (for callers that want to look at
// p.grad after synchronize()).  g must have been zeroed by the caller.
__global__ void __launch_bounds__(256)
k3_scatter_dense(float* g, const Pair* pairs,
                 const unsigned int* counts, unsigned int seg_stride, float scale, unsigned int d, int use_atomics,
                 const unsigned int* parity_word, unsigned int parity_stride) {
  pdl_begin(g, pairs, counts, parity_word);
  pairs = parity_base(pairs, parity_word, parity_stride);
  const Pair* seg = pairs + (size_t)blockIdx.y * seg_stride;
  unsigned int n = counts[blockIdx.y];
  if (n > seg_stride) n = seg_stride;
  const unsigned int stride = gridDim.x * blockDim.x;
  for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const Pair e = seg[i];
    if ((unsigned int)e.idx >= d) continue;
    if (use_atomics) atomicAdd(&g[e.idx], e.val * scale);
    else g[e.idx] = e.val * scale;
  }
}

// Momentum correction (distributed_optimizer.py:81-88 in the reference, off by default there): the
// velocity, not the raw gradient, is what gets sparsified.  v = m*v + g; g = v, over a whole merged
// group in one pass (the reference does it per parameter tensor inside the gradient hook).
__global__ void __launch_bounds__(kK3Threads, 2)
k3_momentum_correct(float* v, float* g, float m, long long d) {
  pdl_begin(v, g);
  const unsigned int mis = (unsigned int)((reinterpret_cast<uintptr_t>(g) >> 2) & 3u);
  long long head = mis ? (4 - mis) : 0;
  if (head > d) head = d;
  const long long nvec = (d - head) >> 2;
  const long long tail0 = head + (nvec << 2);
  float4* v4 = reinterpret_cast<float4*>(v + head);
  float4* g4 = reinterpret_cast<float4*>(g + head);
  const long long stride = (long long)gridDim.x * kK3Threads;
  for (long long i = (long long)blockIdx.x * kK3Threads + threadIdx.x; i < nvec; i += stride) {
    float4 a = v4[i];
    const float4 b = g4[i];
    a.x = fmaf(m, a.x, b.x); a.y = fmaf(m, a.y, b.y); a.z = fmaf(m, a.z, b.z); a.w = fmaf(m, a.w, b.w);
    v4[i] = a;
    g4[i] = a;
  }
  if (blockIdx.x == 0) {
    const long long nscalar = head + (d - tail0);
    for (long long j = threadIdx.x; j < nscalar; j += kK3Threads) {
      const long long i = j < head ? j : tail0 + (j - head);
      const float a = fmaf(m, v[i], g[i]);
      v[i] = a;
      g[i] = a;
    }
  }
}

}  // namespace gtk

using namespace gtk;

static int dense_grid(long long d) {
  const DeviceInfo* di = gtk_device_info();
  const int sms = di ? di->sms : 148;
  long long need = (d / 4 + 2ll * kK3Threads - 1) / (2ll * kK3Threads);
  long long grid = (long long)sms * 2;
  if (need < grid) grid = need > 0 ? need : 1;
  return (int)grid;
}

extern "C" int gtk_k3_dense(float* p, float* buf, const float* g, const float* coef, float scale,
                            long long d, float lr, const float* lr_ptr, float momentum, float dampening,
                            float weight_decay, int nesterov, int first_step, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (d <= 0) return GTK_ERR_ARG;
  const bool has_buf = momentum != 0.f && buf != nullptr;
  const bool has_g = g != nullptr;
  if (!has_g && !has_buf && weight_decay == 0.f) return GTK_OK;  // nothing to do
  const uintptr_t a = reinterpret_cast<uintptr_t>(p) & 15u;
  if ((has_buf && (reinterpret_cast<uintptr_t>(buf) & 15u) != a) ||
      (has_g && (reinterpret_cast<uintptr_t>(g) & 15u) != a))
    return GTK_ERR_ARG;
  SgdHyper h{lr_ptr, lr, momentum, dampening, weight_decay, nesterov, first_step};
  const int grid = dense_grid(d);
  cudaError_t e;
  if (has_g && has_buf) e = launch_pdl(k3_dense<true, true>, grid, kK3Threads, stream, p, buf, g, coef, scale, d, h);
  else if (has_g) e = launch_pdl(k3_dense<true, false>, grid, kK3Threads, stream, p, p, g, coef, scale, d, h);
  else if (has_buf) e = launch_pdl(k3_dense<false, true>, grid, kK3Threads, stream, p, buf, p, coef, scale, d, h);
  else e = launch_pdl(k3_dense<false, false>, grid, kK3Threads, stream, p, p, p, coef, scale, d, h);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}

// n_pairs: how many pairs may be read from `pairs` on (0: only the valid ones).  max_count: as many of them as a list
// has entries (0: not known); lists that are longer all the same are worked off too.
extern "C" int gtk_k3_sparse(float* p, float* buf, const void* pairs, const unsigned int* counts,
                             unsigned int nseg, unsigned int seg_stride, const float* coef,
                             float scale, unsigned int d, float lr, const float* lr_ptr, float momentum,
                             float dampening, float weight_decay, int nesterov, int first_step,
                             int use_atomics, unsigned int* bad_index_count,
                             const unsigned int* parity_word, unsigned int parity_stride,
                             unsigned long long n_pairs, unsigned int max_count, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (nseg == 0 || seg_stride == 0) return GTK_ERR_ARG;
  SgdHyper h{lr_ptr, lr, momentum, dampening, weight_decay, nesterov, first_step};
  const unsigned int length = max_count && max_count < seg_stride ? max_count : seg_stride;
  const unsigned int most = kSparseMaxBlocks / nseg;
  unsigned int blocks = (length + kSparseThreads - 1u) / kSparseThreads;
  if (blocks > most) blocks = most ? most : 1u;
  // Behind a large exchange (a cooperative kernel, which cannot overlap) an ordinary launch: there the overlapped
  // one made the next exchange start 2 us later (57.3 against 55.4 us per exchange + update at 2 x 66 000).
  const bool overlap = parity_word == nullptr || seg_stride <= kLLMaxK;
  const int ahead = (unsigned long long)nseg * length <= kSparseAhead &&
                    n_pairs >= (unsigned long long)nseg * seg_stride + (parity_word ? parity_stride : 0u);
  const cudaError_t e = launch_pdl_if(overlap, k3_sparse, dim3(blocks, nseg), kSparseThreads, stream, p, buf, (const Pair*)pairs, counts,
                                      seg_stride, coef, scale, d, h, use_atomics, bad_index_count, parity_word, parity_stride, ahead);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}

extern "C" int gtk_k3_scatter_dense(float* g, const void* pairs, const unsigned int* counts,
                                    unsigned int nseg, unsigned int seg_stride, float scale,
                                    long long d, int use_atomics, const unsigned int* parity_word,
                                    unsigned int parity_stride, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (cudaMemsetAsync(g, 0, (size_t)d * sizeof(float), stream) != cudaSuccess) return GTK_ERR_CUDA;
  if (nseg == 0 || seg_stride == 0) return GTK_OK;
  unsigned int blocks = (seg_stride + 255u) / 256u;
  if (blocks > 1184u) blocks = 1184u;
  const cudaError_t e = launch_pdl(k3_scatter_dense, dim3(blocks, nseg), 256, stream, g, (const Pair*)pairs, counts,
                                   seg_stride, scale, (unsigned int)d, use_atomics, parity_word, parity_stride);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}

extern "C" int gtk_k3_momentum_correct(float* v, float* g, float momentum, long long d, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (d <= 0 || !v || !g) return GTK_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(v) & 15u) != (reinterpret_cast<uintptr_t>(g) & 15u)) return GTK_ERR_ARG;
  const cudaError_t e = launch_pdl(k3_momentum_correct, dense_grid(d), kK3Threads, stream, v, g, momentum, d);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}
