// Device memory of the contexts: allocations that, where the device has no
// room, ask again once the contexts' memory pools have given back what they
// cache. A pool keeps released scenes (pt_context::kPoolKeep), which neither
// the driver nor another pool can take from it.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ptd {

// `alloc()`; where it fails for want of memory, `trim()` and `alloc()` once
// more.
template <class Alloc, class Trim>
cudaError_t alloc_or_trim(Alloc &&alloc, Trim &&trim) {
  const cudaError_t e = alloc();
  if (e != cudaErrorMemoryAllocation) return e;
  trim();
  return alloc();
}

// The process's pools, each with the stream that its memory is freed on.
// A pool is unregistered before it or its stream is destroyed.
void register_pool(int device, cudaMemPool_t pool, cudaStream_t stream);
void unregister_pool(cudaMemPool_t pool);
// Every pool of the current device gives its cached memory back (waits for
// the pools' streams).
void trim_pools();

// Device memory for scenes, their trees and build scratch: from `pool`
// (stream-ordered; the context's, see pt_context::pool), else from the
// device's default pool on `stream`, else synchronously. Asks again after
// trim_pools; a failure leaves no error for a later launch to report.
cudaError_t device_alloc(void **p, uint64_t bytes, cudaStream_t stream, cudaMemPool_t pool);
// The same for memory that cudaFree returns.
inline cudaError_t device_malloc(void **p, uint64_t bytes) { return device_alloc(p, bytes, nullptr, nullptr); }

}  // namespace ptd
