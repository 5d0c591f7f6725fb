// flow_f32_inv.cu -- inverse instantiations of the fused FP32 flow pass.
#include "flow_f32_kernel.cuh"

namespace fmc {

int launch_flow_f32_inv(const FlowF32Args& a, int R, size_t bytes, cudaStream_t st) {
  return R == 64 ? launch_r<64, true, false>(a, bytes, st) : launch_r<16, true, false>(a, bytes, st);
}

}  // namespace fmc
