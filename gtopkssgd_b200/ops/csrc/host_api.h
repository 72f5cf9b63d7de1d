// C ABI of libgtopk_b200.so.  Every entry point takes raw device pointers and a
// CUDA stream handle, enqueues work on that stream and returns without
// synchronising.  Return value: GTK_OK or a negative GTK_ERR_* code.
// Device-side failures (a wait that ran out, a full list) are reported through
// the status word of the control block, which the caller reads when it wants to.
#pragma once
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum {
  GTK_OK = 0,
  GTK_ERR_ARG = -1,
  GTK_ERR_CUDA = -2,
  GTK_ERR_UNSUPPORTED = -3,
};

// Persistent per-group selection state (device memory, 64 bytes, zero except tau = +inf at first).
typedef struct K1State {
  float tau;                 // candidate threshold of the next stream pass (+inf: none yet)
  unsigned int n_sel;        // pairs written by the last select
  unsigned int n_cand;       // candidates seen by the last stream pass (may exceed the list size)
  unsigned int fallback;     // 1 if the last call took the exact dense path
  unsigned int n_fallbacks;  // running count of exact dense passes
  unsigned int n_calls;      // running count of calls
  float kth_mag;             // exact k-th magnitude of the last call
  unsigned int stream_calls; // calls whose stream pass has begun
  unsigned int aimed;        // candidates that tau was aimed at (0: tau is no prediction)
  float slack;               // decaying maximum of |log(candidates found / aimed)|
  float alpha;               // smoothed tail exponent (0: not measured yet)
  unsigned int reserved[5];
} K1State;

typedef struct DeviceInfo {
  int device;
  int sms;
  int coop;
  int cluster;
} DeviceInfo;

// A list of device addresses, in host memory.
typedef struct gtk_addresses {
  const unsigned long long* p;
  unsigned int n;
} gtk_addresses;

const DeviceInfo* gtk_device_info(void);
void gtk_count_launch(int n);
long long gtk_launch_count(void);
void gtk_reset_launch_count(void);
unsigned long long gtk_ctrl_bytes(void);
unsigned long long gtk_k1state_bytes(void);
const char* gtk_last_cuda_error(void);

// ---- launches (each file documents its own) ----
int gtk_k1_pick_is_wide(long long d, unsigned int k, int compress);
int gtk_k1_select(const float* g, float* r, const float* g_scale, long long d, unsigned int k,
                  void* cand, unsigned int cap, void* sel, void* state, void* ctrl,
                  float target_ratio, unsigned long long limit_ns, void* stream);
int gtk_k1_select_segments(gtk_addresses grads, const unsigned int* segments, float* r, long long d, unsigned int k,
                           void* cand, unsigned int cap, void* sel, void* state, void* ctrl, float target_ratio,
                           unsigned long long limit_ns, void* stream);
int gtk_k1_compress(float* g, float* r, long long d, unsigned int k, void* cand, unsigned int cap, void* sel,
                    void* state, void* ctrl, float target_ratio, unsigned long long limit_ns, long long* idx_out,
                    float* val_out, void* stream);
int gtk_k2_exchange(const void* ranks_dev, unsigned int nranks, unsigned int rank_base, unsigned int P,
                    unsigned int k, unsigned int kcap, unsigned int d, unsigned int nctas,
                    unsigned long long limit_ns, int use_cluster, void* stream);
int gtk_k2t_allgather(const void* ranks_dev, unsigned int nranks, unsigned int rank_base,
                      unsigned int P, unsigned int k, unsigned int kcap, unsigned int work_cap, unsigned int d,
                      int reselect, void* seg_counts, unsigned int nctas, unsigned long long limit_ns, void* stream);
int gtk_k3_dense(float* p, float* buf, const float* g, const float* coef, float scale, long long d, float lr,
                 const float* lr_ptr, float momentum, float dampening, float weight_decay, int nesterov,
                 int first_step, void* stream);
int gtk_k3_sparse(float* p, float* buf, const void* pairs, const unsigned int* counts, unsigned int nseg,
                  unsigned int seg_stride, const float* coef, float scale, unsigned int d, float lr,
                  const float* lr_ptr, float momentum, float dampening, float weight_decay, int nesterov,
                  int first_step, int use_atomics, unsigned int* bad_index_count, const unsigned int* parity_word,
                  unsigned int parity_stride, unsigned long long n_pairs, unsigned int max_count, void* stream);
int gtk_k3_scatter_dense(float* g, const void* pairs, const unsigned int* counts, unsigned int nseg,
                         unsigned int seg_stride, float scale, long long d, int use_atomics,
                         const unsigned int* parity_word, unsigned int parity_stride, void* stream);
int gtk_k3_momentum_correct(float* v, float* g, float momentum, long long d, void* stream);
int gtk_k4_sumsq_dense(const float* x, long long d, void* state, void* stream);
int gtk_k4_sumsq_pairs(const void* pairs, const unsigned int* counts, unsigned int nseg, unsigned int seg_stride,
                       void* state, const unsigned int* parity_word, unsigned int parity_stride, void* stream);
int gtk_k4_finalize(void* state, float scale, float max_norm, float* coef_out, void* stream);
int gtk_k5_top1(const float* logits, const long long* target, int rows, int classes, float scale, float* out,
                void* stream);

#ifdef __cplusplus
}
#endif
