// K5: top-1 accuracy of a batch of logits, in per cent.
//
// The training loop reports it every iteration (dl_trainer.py:566-568 in the
// reference: topk, transpose, compare, sum, scale); as library calls that were
// eight launches on a few kilobytes, 0.1 ms of host time of a 4.4 ms ResNet-20
// iteration.  One CTA, a warp per row: the arrays are small (64 x 1000 floats at
// most in the named configurations, 3 us).
#include "common.cuh"
#include "host_api.h"
#include "launch.cuh"

namespace gtk {

constexpr int kK5Threads = 1024;

// NaN counts as the largest value, as in torch.topk; of equal values the first one.
__device__ __forceinline__ bool better(float a, int ia, float b, int ib) {
  if (isnan(a) != isnan(b)) return isnan(a);
  if (a != b && !isnan(a)) return a > b;
  return ia < ib;
}

__global__ void __launch_bounds__(kK5Threads)
k5_top1(const float* logits, const long long* target, int rows, int classes, float scale, float* out) {
  __shared__ int hits;
  if (threadIdx.x == 0) hits = 0;
  __syncthreads();
  pdl_begin(logits, target);
  int mine = 0;
  for (int row = (int)(threadIdx.x >> 5); row < rows; row += kK5Threads / 32) {
    const float* x = logits + (size_t)row * classes;
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int c = (int)lane_id(); c < classes; c += 32)
      if (at == 0x7fffffff || better(x[c], c, best, at)) {
        best = x[c];
        at = c;
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float b = __shfl_xor_sync(0xffffffffu, best, o);
      const int ib = __shfl_xor_sync(0xffffffffu, at, o);
      if (ib != 0x7fffffff && (at == 0x7fffffff || better(b, ib, best, at))) {
        best = b;
        at = ib;
      }
    }
    mine += (long long)at == target[row] ? 1 : 0;
  }
  if (lane_id() == 0 && mine) atomicAdd(&hits, mine);
  __syncthreads();
  if (threadIdx.x == 0) *out = (float)hits * scale;
}

}  // namespace gtk

using namespace gtk;

// out = (rows whose first largest logit is at target[row]) * scale
extern "C" int gtk_k5_top1(const float* logits, const long long* target, int rows, int classes, float scale, float* out,
                           void* stream_) {
  if (rows <= 0 || classes <= 0) return GTK_ERR_ARG;
  const cudaError_t e = launch_pdl(k5_top1, 1, kK5Threads, (cudaStream_t)stream_, logits, target, rows, classes, scale, out);
  gtk_count_launch(1);
  return e == cudaSuccess ? GTK_OK : GTK_ERR_CUDA;
}
