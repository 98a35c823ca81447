#include "device_mem.h"

#include <algorithm>
#include <mutex>
#include <vector>

namespace ptd {

namespace {

struct Pools {
  struct Entry {
    int device;
    cudaMemPool_t pool;
    cudaStream_t stream;
  };
  std::mutex m;
  std::vector<Entry> all;
};
Pools &pools() {
  static Pools p;
  return p;
}

}  // namespace

void register_pool(int device, cudaMemPool_t pool, cudaStream_t stream) {
  std::lock_guard<std::mutex> lock(pools().m);
  pools().all.push_back({device, pool, stream});
}

void unregister_pool(cudaMemPool_t pool) {
  std::lock_guard<std::mutex> lock(pools().m);
  std::vector<Pools::Entry> &all = pools().all;
  all.erase(std::remove_if(all.begin(), all.end(), [&](const Pools::Entry &e) { return e.pool == pool; }), all.end());
}

void trim_pools() {
  int device = 0;
  if (cudaGetDevice(&device) == cudaSuccess) {
    std::lock_guard<std::mutex> lock(pools().m);
    for (const Pools::Entry &e : pools().all)
      if (e.device == device) {
        // Memory goes back once the frees before it in the stream are done.
        cudaStreamSynchronize(e.stream);
        cudaMemPoolTrimTo(e.pool, 0);
      }
  }
  cudaGetLastError();
}

cudaError_t device_alloc(void **p, uint64_t bytes, cudaStream_t stream, cudaMemPool_t pool) {
  return alloc_or_trim(
      [&] {
        const cudaError_t e = pool     ? cudaMallocFromPoolAsync(p, bytes, pool, stream)
                              : stream ? cudaMallocAsync(p, bytes, stream)
                                       : cudaMalloc(p, bytes);
        if (e != cudaSuccess) cudaGetLastError();
        return e;
      },
      [] { trim_pools(); });
}

}  // namespace ptd
