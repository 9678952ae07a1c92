// Dynamic shared memory above the 48 KB default: raising a kernel's limit.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <map>
#include <mutex>
#include <utility>

namespace llmctl {

// Raises cudaFuncAttributeMaxDynamicSharedMemorySize of a kernel on the current device to at least `bytes`.  The limit belongs to the
// kernel and the device, and the runtime call lowers it just as well: a thread that set it for a smaller size would make the launches of
// others fail.  So the limits set so far stand in one table for all threads and only grow.  The runtime call costs about as much host
// time as a quarter of a launch; what a thread has once seen raised it looks up without the lock.
inline cudaError_t raise_smem_limit(const void* kernel, int bytes) {
  struct Entry {
    const void* f;
    int device, bytes;
  };
  static thread_local Entry seen[64] = {};
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> limits;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  Entry& at = seen[(reinterpret_cast<uintptr_t>(kernel) >> 4) & 63];
  if (at.f == kernel && at.device == device && at.bytes >= bytes) return cudaSuccess;
  std::lock_guard<std::mutex> hold(mu);
  int* limit;
  try {
    limit = &limits[std::make_pair(kernel, device)];
  } catch (...) {
    return cudaErrorMemoryAllocation;
  }
  if (*limit < bytes) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    *limit = bytes;
  }
  at = Entry{kernel, device, *limit};
  return cudaSuccess;
}

template <typename Kernel>
inline cudaError_t allow_smem(Kernel kernel, int bytes) {
  return raise_smem_limit(reinterpret_cast<const void*>(kernel), bytes);
}

}  // namespace llmctl
