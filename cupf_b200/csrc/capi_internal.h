// capi_internal.h — error plumbing shared by the library's C ABI translation units.
#pragma once

#include <cuda_runtime.h>

#include <initializer_list>

#include "../../include/cupf.h"

// Records a per-thread message (returned by cupf_last_error) and returns st.
cupf_status cupf_fail(cupf_status st, const char* fmt, ...);

#define CK(call)                                                                       \
  do {                                                                                 \
    cudaError_t e_ = (call);                                                           \
    if (e_ != cudaSuccess)                                                             \
      return cupf_fail(e_ == cudaErrorMemoryAllocation ? CUPF_ERR_OOM : CUPF_ERR_CUDA, \
                       "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_),         \
                       __FILE__, __LINE__);                                            \
  } while (0)

// Device buffers that a call allocates together: all of them or, where one does not
// fit, none (a later call then tries again; nothing is left half set up).
struct DeviceBuffer {
  void** p;
  size_t bytes;
};
inline cudaError_t malloc_together(std::initializer_list<DeviceBuffer> bufs) {
  cudaError_t e = cudaSuccess;
  for (const DeviceBuffer& b : bufs) *b.p = nullptr;
  for (const DeviceBuffer& b : bufs)
    if (e == cudaSuccess) e = cudaMalloc(b.p, b.bytes);
  if (e == cudaSuccess) return e;
  for (const DeviceBuffer& b : bufs) {
    if (*b.p) cudaFree(*b.p);
    *b.p = nullptr;
  }
  cudaGetLastError();  // reported by the return value, not by the next launch's check
  return e;
}

// Programmatic dependent launch of a step kernel: its blocks are set up while the last
// ones of the kernel before it in the stream run, and wait for that kernel's end
// (cudaGridDependencySynchronize) before they touch global memory.
template <class... P, class... A>
cudaError_t launch_dependent(cudaStream_t stream, dim3 grid, dim3 block, size_t smem,
                             void (*kernel)(P...), const A&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
