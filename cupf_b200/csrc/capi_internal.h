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

// Frees the slot maps of one of the process's simulations on the current device, once
// the steps queued on it are done; false where none is left to free.  The maps are
// optional memory: a simulation without them merges every cell every step, with the
// same results.
bool release_slot_maps();
// Bytes that release_slot_maps could free on `device`.
size_t held_slot_map_bytes(int device);

// An allocation that the slot maps give way to: run again after each release while the
// device is out of memory.  A failure is reported by the return value, not by the next
// launch's error check too.
template <class F>
cudaError_t with_room(F&& allocate) {
  cudaError_t e = allocate();
  while (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (!release_slot_maps()) break;
    e = allocate();
  }
  return e;
}
template <class T>
cudaError_t device_malloc(T** p, size_t bytes) {
  return with_room([&] { return cudaMalloc((void**)p, bytes); });
}

// Device buffers that a call allocates together: all of them or, where one does not
// fit, none (a later call then tries again; nothing is left half set up).
struct DeviceBuffer {
  void** p;
  size_t bytes;
};
inline cudaError_t malloc_together(std::initializer_list<DeviceBuffer> bufs,
                                   bool make_room = true) {
  cudaError_t e = cudaSuccess;
  for (const DeviceBuffer& b : bufs) *b.p = nullptr;
  for (const DeviceBuffer& b : bufs)
    if (e == cudaSuccess) e = make_room ? device_malloc(b.p, b.bytes) : cudaMalloc(b.p, b.bytes);
  if (e == cudaSuccess) return e;
  for (const DeviceBuffer& b : bufs) {
    if (*b.p) cudaFree(*b.p);
    *b.p = nullptr;
  }
  cudaGetLastError();
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
