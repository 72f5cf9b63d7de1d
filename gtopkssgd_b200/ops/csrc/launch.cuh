// Launches that overlap with the end of the kernel before them.
//
// A kernel that depends on its predecessor in the stream normally starts 1.5 to
// 3 us after it has ended (measured on B200, chains of short kernels: 2.06 us per
// empty kernel, 4.10 us for a body of 2.04 us, cooperative launches alike).  With
// programmatic stream serialization the CTAs are placed while the predecessor
// drains and griddepcontrol.wait lets them go: 0.6 to 0.9 us on top of the body.
// Every kernel launched here executes pdl_begin() before its first access to
// global memory, so it sees all of its predecessor's results; the early trigger
// inside lets its own successor be placed in turn.
#pragma once
#include <cuda_runtime.h>

namespace gtk {

// The pointers that the kernel reads through pass an empty asm statement behind the wait, so that the
// compiler cannot take a load ahead of it (a memory clobber alone does not bind read-only accesses).
template <typename... P>
__device__ __forceinline__ void pdl_begin(P*&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  ((void)([](P*& q) { asm volatile("" : "+l"(q)::"memory"); }(p)), ...);
}

// overlap = false: an ordinary launch of the same kernel.
template <typename... K, typename... A>
inline cudaError_t launch_pdl_if(bool overlap, void (*kernel)(K...), dim3 grid, dim3 block, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}
template <typename... K, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(K...), dim3 grid, dim3 block, cudaStream_t stream, A&&... args) {
  return launch_pdl_if(true, kernel, grid, block, stream, static_cast<A&&>(args)...);
}

}  // namespace gtk
