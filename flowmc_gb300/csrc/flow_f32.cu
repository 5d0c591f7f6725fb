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

bool flow_f32_tile_fits(const FlowGeom& g, int R, size_t* bytes) {
  FlowF32Args a{};
  return flow_f32_smem(g, R, a, *bytes);
}

// The fastest way through a forward or inverse pass: 64 or 16 rows per CTA of
// the fused kernel, or 0 for the launches per layer (the same bits all three).
// 16-row tiles win on few rows of narrow conditioners (one launch instead of
// five per layer), 64-row tiles on many rows where two CTAs share an SM, and the
// layered 64 x 64 GEMM tiles where a row tile's serial walk over all weights is
// long (wide layers, many coordinate groups) or a lone CTA per SM leaves its
// splines uncovered. Where the lines lie depends on all of the sizes, so each way
// is estimated in microseconds per layer from the counts that drive it:
//   S   stages (16 inputs x one tile of outputs) of the conditioner
//   G   coordinate groups of its last Linear (splines between products)
//   t   row tiles on the fullest SM, r the rounds they run in
// with coefficients fitted to 630 measured calls (GB300; 5 to 500 dims, 16 to 768
// units, 4 to 12 bins, 16 to 100,000 rows, 4 layers), which they reproduce
// within 10 % (16 and 64 rows) and 17 % (layers) for nine calls in ten. The fused
// kernel has to look a tenth faster; the choice is then within 1 % of the fastest
// of the three on average, at worst 28 % behind it, and at worst 14 % behind the
// layers. Taking the fused kernel wherever it fits had cost, against the
// layers, in us: 32-D, 10 bins, 512 units, 100,000 rows 14,341 -> 24,452; 128-D,
// 12 bins, 768 units, 16 rows 551 -> 2,873; 128-D, 4 bins, 16 units, 100,000
// rows 1,409 -> 2,273.
int flow_f32_route(const FlowGeom& g, int64_t n) {
  const FlowShape s = flow_shape(g);
  const double sms = sm_count();
  double S = 0, G = 0, steps = 0, macs = 0, raw = 0;   // means over the two layer parities
  for (int l = 0; l < 2; ++l)
    for (int i = 0; i <= g.nh; ++i) {
      const int in = s.in(l, i), out = s.out(l, i), tc = s.tile_cols(i);
      const int tiles = (out + tc - 1) / tc, ks = (in + kFlowBK - 1) / kFlowBK;
      S += 0.5 * tiles * ks;
      steps += 0.5 * ks;
      macs += 0.5e-6 * ((out + 63) / 64 * 64) * (ks * kFlowBK);   // a 64 x 64 GEMM's, padded, in millions
      if (i == g.nh) {
        G += 0.5 * tiles;
        raw += 0.5e-6 * out;
      }
    }
  double best = 0.9 * (28.9 + 0.787 * steps + (double)n * (0.0601 * macs + 1.835 * raw + 0.88e-3));
  int route = 0;
  for (int R = 16; R <= 64; R += 48) {
    FlowF32Args a{};
    size_t bytes = 0;
    if (!flow_f32_smem(g, R, a, bytes)) continue;
    const double t = ceil(ceil((double)n / R) / sms);
    const double r = ceil(t / (2 * (bytes + 1024) <= 228 * 1024 ? 2 : 1));
    const double est = R == 16 ? 5.4 + r * (1.5 + 0.256 * S + 1.41 * G) + t * (0.256 * S + 0.05 * G)
                               : 6.6 + r * (7.6 + 0.578 * S + 1.69 * G) + t * (0.473 * S + 0.101 * g.d);
    if (est < best) {
      best = est;
      route = R;
    }
  }
  return route;
}

int flow_f32_pass(const FlowF32Call& c, const FlowGeom& g, int R, cudaStream_t st) {
  if (c.n <= 0) return FMC_OK;
  FlowF32Args a{};
  size_t bytes = 0;
  if (!flow_f32_smem(g, R, a, bytes)) {
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
  a.tiles = (c.n + R - 1) / R;
  if (c.acts != nullptr) return launch_flow_f32_save(a, R, bytes, st);
  return c.inverse ? launch_flow_f32_inv(a, R, bytes, st) : launch_flow_f32_fwd(a, R, bytes, st);
}

}  // namespace fmc
