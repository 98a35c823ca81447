// k_wf_shade for plain materials.
#include "wavefront_shade.cuh"

namespace ptd {

cudaError_t set_shade_plain_tables(const float *sheen_lut) {
  return cudaMemcpyToSymbol(g_sheen_lut, sheen_lut, sizeof(float) * SHEEN_LUT_COS * SHEEN_LUT_ROUGH);
}

void launch_wf_shade_plain(const WaveBuffers &w, uint32_t it, int num_sms, cudaStream_t st) {
  constexpr int kThreads = 256, kBlocks = 2;
  k_wf_shade<kThreads, kBlocks, true><<<num_sms * kBlocks * 2, kThreads, 0, st>>>(w, it);
}

}  // namespace ptd
