// The wavefront's traversal kernels and their launchers, in a translation
// unit of their own (the shading kernels take minutes to compile).
#include <algorithm>

#include "kernels.h"
#include "per_device.h"
#include "wavefront_trace.cuh"

namespace ptd {

// The traversal kernels are persistent: exactly the blocks that fit at once.
// Index [t][o]: t = 0 the 256-thread instantiations, 1 the 128-thread ones;
// o = 1 the four-child-only ones.
struct TraceBlocks {
  int ext[2][2], sh[2][2];  // per SM
};

static void query_trace_blocks(int device, TraceBlocks &out) {
  // The traversal kernels are register-bound at 1,024 threads per SM and
  // need shared memory only for their stacks and counts (19 words a thread,
  // 76 KB an SM): ask for the smallest shared-memory carveout that holds
  // those blocks, so the rest of the SM's on-chip memory serves as L1 for
  // nodes and triangle records.
  int smem_sm = 0;
  if (cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device) != cudaSuccess) smem_sm = 0;
  cudaGetLastError();
  auto q = [smem_sm](int &v, const void *fn, int threads) {
    const long shared = threads == 256 ? (long)sizeof(TraceShared<256>) : (long)sizeof(TraceShared<128>);
    if (smem_sm > 0) {
      const long need = (1024L / threads) * (shared + 1024L);
      const int pct = (int)std::min(100L, (need * 100L + smem_sm - 1) / smem_sm + 1);
      if (cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct) != cudaSuccess)
        cudaGetLastError();
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, fn, threads, 0) != cudaSuccess || v < 1) v = 1;
  };
  q(out.ext[0][0], (const void *)k_wf_extend<256, false>, 256);
  q(out.ext[0][1], (const void *)k_wf_extend<256, true>, 256);
  q(out.sh[0][0], (const void *)k_wf_shadow<256, false>, 256);
  q(out.sh[0][1], (const void *)k_wf_shadow<256, true>, 256);
  q(out.ext[1][0], (const void *)k_wf_extend<128, false>, 128);
  q(out.ext[1][1], (const void *)k_wf_extend<128, true>, 128);
  q(out.sh[1][0], (const void *)k_wf_shadow<128, false>, 128);
  q(out.sh[1][1], (const void *)k_wf_shadow<128, true>, 128);
}

// The current device's table. Contexts of several threads may ask for it at
// once; the carveout is an attribute of each device's copy of the kernels.
static const TraceBlocks &trace_blocks() {
  static PerDevice<TraceBlocks> blocks;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) cudaGetLastError();
  return blocks.get(device, [device](TraceBlocks &b) { query_trace_blocks(device, b); });
}

// The traversal launches of one bounce iteration: block size and node
// layout choose the instantiation.
template <int kThreads>
static void launch_extend(const WaveBuffers &w, uint32_t it, DevCounters *ctr, uint32_t grid, bool only4, cudaStream_t st) {
  if (only4)
    k_wf_extend<kThreads, true><<<grid, kThreads, 0, st>>>(w, it, ctr);
  else
    k_wf_extend<kThreads, false><<<grid, kThreads, 0, st>>>(w, it, ctr);
}
template <int kThreads>
static void launch_shadow(const WaveBuffers &w, uint32_t it, DevCounters *ctr, uint32_t grid, bool only4, cudaStream_t st) {
  if (only4)
    k_wf_shadow<kThreads, true><<<grid, kThreads, 0, st>>>(w, it, ctr);
  else
    k_wf_shadow<kThreads, false><<<grid, kThreads, 0, st>>>(w, it, ctr);
}

void prepare_trace_kernels() { trace_blocks(); }

void launch_wf_extend(const WaveBuffers &w, uint32_t it, DevCounters *ctr, int num_sms, cudaStream_t st) {
  const bool t128 = w.trav_threads == 128, only4 = (w.all_wide & WIDE_EXTENSION) != 0;
  const uint32_t grid = (uint32_t)(num_sms * trace_blocks().ext[t128 ? 1 : 0][only4 ? 1 : 0]);
  if (t128)
    launch_extend<128>(w, it, ctr, grid, only4, st);
  else
    launch_extend<256>(w, it, ctr, grid, only4, st);
}

void launch_wf_shadow(const WaveBuffers &w, uint32_t it, DevCounters *ctr, int num_sms, cudaStream_t st) {
  const bool t128 = w.trav_threads == 128, only4 = (w.all_wide & WIDE_SHADOW) != 0;
  const uint32_t grid = (uint32_t)(num_sms * trace_blocks().sh[t128 ? 1 : 0][only4 ? 1 : 0]);
  if (t128)
    launch_shadow<128>(w, it, ctr, grid, only4, st);
  else
    launch_shadow<256>(w, it, ctr, grid, only4, st);
}

}  // namespace ptd
