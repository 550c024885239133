// Backward scan kernels for d_state 16 and __nv_bfloat16 activations.
#include "sscan_bwd16_launch.cuh"

namespace mb200 {

int bwd16_launch_bf16(const SscanBwdParams& p, bool carry_only, cudaStream_t st) { return bwd16_launch<__nv_bfloat16>(p, carry_only, st); }
int bwd16_status_bf16() { return bwd16_status(); }

}  // namespace mb200
