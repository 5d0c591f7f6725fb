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
  // training (forward, FLOW_OUT_LOGP), both or neither: [L + 1, n, d] layer
  // inputs and the output, and the activations flow_f32_grad reads
  float* save;
  float* acts;
};

// whether a tile of R rows fits in shared memory, and the bytes it takes
bool flow_f32_tile_fits(const FlowGeom& g, int R, size_t* bytes);
// rows per CTA of a forward or inverse pass over n rows; 0: the launches per layer are faster
int flow_f32_route(const FlowGeom& g, int64_t n);
// all layers over c.n rows in one launch of R-row tiles
int flow_f32_pass(const FlowF32Call& c, const FlowGeom& g, int R, cudaStream_t st);

// floats of split-K partials the FP32 weight gradients may use (they bound the
// number of slices, and with it the order of the sums)
int64_t kouter_part_floats(const FlowGeom& g);
// The loss gradient from a forward pass that left `save` and `acts`
// (flow_f32_bwd.cu): how n rows train -- `tile` rows per CTA of both passes and per
// tile of the saved activations (0 where the flow does not fit: hidden widths
// and conditioning block up to 128), and whether that is faster than the
// launches per layer --, floats of its workspace (the activations first), and the
// gradient itself into grad [n_params].
struct FlowGradRoute {
  int tile;
  bool faster;
};
FlowGradRoute flow_f32_grad_route(const FlowGeom& g, int64_t n);
int64_t flow_f32_grad_floats(const FlowGeom& g, int64_t n);
int flow_f32_grad(const FlowGeom& g, const float* theta, const float* aux, int64_t n, const float* save, float* ws,
                  float* grad, cudaStream_t st);

}  // namespace fmc
