// A kernel's limit of dynamic shared memory, which belongs to a device: raised at its first launch on each.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

namespace dcpk {

// `raised`: of one kernel, a bit per device on which the limit has been raised (devices from 64 on: on every call).
// Two threads that come at once both raise it, which does no harm.
template <typename K>
inline cudaError_t raise_smem_limit(K kernel, int bytes, std::atomic<uint64_t>& raised) {
  int device = 0;
  const cudaError_t found = cudaGetDevice(&device);
  if (found != cudaSuccess) return found;
  const uint64_t bit = device < 64 ? uint64_t(1) << device : 0;
  if (raised.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  const cudaError_t rc =
      cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (rc == cudaSuccess) raised.fetch_or(bit, std::memory_order_relaxed);
  return rc;
}

}  // namespace dcpk
