// flow_f32.h -- entry of the fused FP32 flow passes (flow_f32.cu).
#pragma once
#include "flow.cuh"

namespace fmc {

enum FlowIn : int { FLOW_IN_ROWS = 0, FLOW_IN_DATA = 1, FLOW_IN_BASE = 2 };     // as given; standardised; base samples
enum FlowOut : int { FLOW_OUT_ROWS = 0, FLOW_OUT_LOGP = 1, FLOW_OUT_DATA = 2 };  // rows + log-det; log-density; destandardised

struct FlowF32Call {
  const float* theta;
  const float* aux;
  const float* x;
  const float* z;
  Rng rng;
  int64_t n;
  bool inverse;
  int in_mode, out_mode;
  float* y;
  float* ld;
  float* logp;
  float* save;
};

// whether the flow's row tile fits in shared memory
bool flow_f32_fused(const FlowGeom& g);
// all layers over c.n rows in one launch
int flow_f32_pass(const FlowF32Call& c, const FlowGeom& g, cudaStream_t st);

}  // namespace fmc
