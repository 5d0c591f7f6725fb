// flow_f32.cu -- host side of the fused FP32 flow passes: tile choice and
// shared-memory layout (kernel: flow_f32_kernel.cuh).
#include "flow_f32_kernel.cuh"

namespace fmc {

// pitches and shared memory of a tile of R rows; false if it does not fit
static bool flow_f32_smem(const FlowGeom& g, int R, FlowF32Args& a, size_t& bytes) {
  int hm = 1;
  for (int i = 0; i < g.nh; ++i) hm = g.H[i] > hm ? g.H[i] : hm;
  const FlowShape s = flow_shape(g);
  a.s = s;
  a.ldx = g.d | 1;                    // rows on different banks for the splines' column reads
  const int ld = R + 4;
  const int cond = ((g.nc_max() + 15) & ~15) * ld;
  a.cond_floats = cond > 32 * R ? cond : 32 * R;
  const int cols = (hm + 15) & ~15, rc = s.dg * s.P;
  a.act_floats = (cols > rc ? cols : rc) * ld;
  const int stages = R >= 64 ? FlowTile<64>::ST : FlowTile<16>::ST;
  bytes = sizeof(float) * ((size_t)R * a.ldx + a.cond_floats + 2 * (size_t)a.act_floats + stages * kFlowStageFloats +
                           256);
  return bytes <= 227 * 1024;
}

int flow_f32_tile(const FlowGeom& g, int64_t n) {
  FlowF32Args a{};
  size_t bytes = 0;
  return n >= 64 * (int64_t)sm_count() && flow_f32_smem(g, 64, a, bytes) ? 64 : 16;
}

bool flow_f32_fused(const FlowGeom& g) {
  FlowF32Args a{};
  size_t b;
  return flow_f32_smem(g, 16, a, b);
}

// rows per CTA: 64 where they fill the SMs and fit in shared memory, else 16
// (fewer rows per CTA and two more warps per row: latency). Measured on GB300,
// 5-D flow 4 x [32, 32]: the 620 rows of a 20-chain global step take 39 CTAs of
// 16 rows; 10,000 rows (157 CTAs of 64) train in 341 us per step, in 16-row tiles
// 425; a remainder launch of 16-row tiles behind whole waves of 64-row ones
// did not pay (100,003 rows of the 32-D flow: 3.72 against 3.64 ms).
int flow_f32_pass(const FlowF32Call& c, const FlowGeom& g, cudaStream_t st) {
  if (c.n <= 0) return FMC_OK;
  FlowF32Args a{};
  size_t bytes = 0;
  const bool wide = flow_f32_tile(g, c.n) == 64 && flow_f32_smem(g, 64, a, bytes);
  if (!wide && !flow_f32_smem(g, 16, a, bytes)) {
    set_error("flow does not fit the fused FP32 kernel");
    return FMC_ERR_UNSUPPORTED;
  }
  a.theta = c.theta;
  a.aux = c.aux;
  a.x = c.x;
  a.z = c.z;
  a.rng = c.rng;
  a.n = c.n;
  a.in_mode = c.in_mode;
  a.out_mode = c.out_mode;
  a.y = c.y;
  a.ld = c.ld;
  a.logp = c.logp;
  a.save = c.save;
  a.acts = c.acts;
  a.tiles = (c.n + (wide ? 64 : 16) - 1) / (wide ? 64 : 16);
  const int R = wide ? 64 : 16;
  if (c.acts != nullptr) return launch_flow_f32_save(a, R, bytes, st);
  return c.inverse ? launch_flow_f32_inv(a, R, bytes, st) : launch_flow_f32_fwd(a, R, bytes, st);
}

}  // namespace fmc
