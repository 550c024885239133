// Backward scan kernels for d_state 16 and float activations.
#include "sscan_bwd16_launch.cuh"

namespace mb200 {

int bwd16_launch_f32(const SscanBwdParams& p, bool carry_only, cudaStream_t st) { return bwd16_launch<float>(p, carry_only, st); }
int bwd16_status_f32() { return bwd16_status(); }

}  // namespace mb200
