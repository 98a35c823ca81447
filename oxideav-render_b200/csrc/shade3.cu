// k_wf_shade at three blocks per SM.
#include "wavefront_shade.cuh"

namespace ptd {

cudaError_t set_shade3_tables(const float *sheen_lut) {
  return cudaMemcpyToSymbol(g_sheen_lut, sheen_lut, sizeof(float) * SHEEN_LUT_COS * SHEEN_LUT_ROUGH);
}

void launch_wf_shade3(const WaveBuffers &w, uint32_t it, uint32_t grid, cudaStream_t st) {
  k_wf_shade<3><<<grid, 128, 0, st>>>(w, it);
}

}  // namespace ptd
