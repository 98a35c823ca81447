// k_wf_shade at four blocks per SM.
#include "wavefront_shade.cuh"

namespace ptd {

cudaError_t set_shade4_tables(const float *sheen_lut) {
  return cudaMemcpyToSymbol(g_sheen_lut, sheen_lut, sizeof(float) * SHEEN_LUT_COS * SHEEN_LUT_ROUGH);
}

void launch_wf_shade4(const WaveBuffers &w, uint32_t it, uint32_t grid, cudaStream_t st) {
  k_wf_shade<4><<<grid, 128, 0, st>>>(w, it);
}

}  // namespace ptd
