// capi_internal.h — error plumbing shared by the library's C ABI translation units.
#pragma once

#include <cuda_runtime.h>

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
