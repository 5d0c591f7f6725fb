// flow_f32_fwd.cu -- forward instantiations of the fused FP32 flow pass.
#include "flow_f32_kernel.cuh"

namespace fmc {

int launch_flow_f32_fwd(const FlowF32Args& a, int R, size_t bytes, cudaStream_t st) {
  return R == 64 ? launch_r<64, false, false>(a, bytes, st) : launch_r<16, false, false>(a, bytes, st);
}

}  // namespace fmc
