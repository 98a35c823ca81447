// k_wf_shade for layered materials at 512 threads per SM.
#include "wavefront_shade.cuh"

namespace ptd {

cudaError_t set_shade4_tables(const float *sheen_lut) {
  return cudaMemcpyToSymbol(g_sheen_lut, sheen_lut, sizeof(float) * SHEEN_LUT_COS * SHEEN_LUT_ROUGH);
}

void launch_wf_shade4(const WaveBuffers &w, uint32_t it, int num_sms, cudaStream_t st) {
  constexpr int kThreads = 512, kBlocks = 1;
  k_wf_shade<kThreads, kBlocks, false><<<num_sms * kBlocks * 2, kThreads, 0, st>>>(w, it);
}

}  // namespace ptd
