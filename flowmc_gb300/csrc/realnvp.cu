// realnvp.cu -- the RealNVP flow (resource/model/nf_model/realNVP.py of flowMC).
//
// A layer is MaskedCouplingLayer(MLPAffine(scale_MLP, shift_MLP, dt), m)
// (realNVP.py:163-176, common.py:127-208):
//   c = x * m,   s = tanh(MLP_s(c)) * dt,   t = MLP_t(c) * dt
//   y = (1 - m) * ((x + t) * exp(s)) + m * x,   log-det = sum (1 - m) * s
// with MLP = Linear(d, H), relu, Linear(H, d). The masks are float leaves of
// the reference model, so optax's weight decay moves them off 0/1; they live
// in aux and every kernel uses the general formula.
//
// Per layer and row block: the first Linears of both MLPs as one GEMM (W1 =
// [W1s; W1t], relu epilogue), the two second Linears as one launch of two GEMMs
// with bias epilogues, then one warp per row applies the coupling, sums the
// log-det and leaves the next layer's masked input. Training keeps every layer's
// masked input, hidden activations and conditioner outputs; the backward is,
// per layer, the coupling adjoint, one launch of the two relu-masked dH GEMMs
// and the dc GEMM, which adds into the input gradient. The weight and bias
// gradients of all layers are formed at the end: one grid of split-row outer
// products with fixed-order slice sums (deterministic), two launches of column
// sums. FP32 SIMT GEMMs throughout (gemm_f32.cuh): RealNVP's MLPs are narrow
// [d, H, d].
//
// Measured on GB300 (32-D, 8 layers, H = 256): loss + gradient of 16,384 rows
// 3.64 -> 1.29 ms (212 launches -> 58; the GEMMs 0.89 ms, the weight gradients
// 0.17 ms = 50 TFLOP/s).
#include "flow.cuh"
#include "gemm_f32.cuh"

namespace fmc {

struct RnvpGeom {
  int d, L, H;
  float dt;
  int64_t off_b1, off_W2s, off_b2s, off_W2t, off_b2t, per_layer, n_params, n_aux;
};

static int rnvp_geom(const FmcRealNVP* f, RnvpGeom& g) {
  FMC_CHECK_ARG(f != nullptr, "flow is NULL");
  FMC_CHECK_ARG(f->n_dim >= 1 && f->n_layers >= 1 && f->n_hidden >= 1, "RealNVP shape d=%d L=%d H=%d", f->n_dim,
                f->n_layers, f->n_hidden);
  g.d = f->n_dim;
  g.L = f->n_layers;
  g.H = f->n_hidden;
  g.dt = f->dt;
  const int64_t d = g.d, H = g.H;
  g.off_b1 = 2 * H * d;
  g.off_W2s = g.off_b1 + 2 * H;
  g.off_b2s = g.off_W2s + d * H;
  g.off_W2t = g.off_b2s + d;
  g.off_b2t = g.off_W2t + d * H;
  g.per_layer = g.off_b2t + d;
  g.n_params = g.per_layer * g.L;
  g.n_aux = 2 * d + 2 + (int64_t)g.L * d;
  return FMC_OK;
}

constexpr int64_t kRnvpChunk = 65536;   // rows per inference chunk
constexpr int kMaxSlices = 64;   // row slices of the weight gradients

static int grid_for(int64_t tot, int per_sm = 8) {
  int64_t b = (tot + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * per_sm;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

static int warp_grid(int64_t rows) {
  int64_t b = (rows + 7) / 8;   // 8 warps per 256-thread block
  const int64_t cap = (int64_t)sm_count() * 16;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

// ------------------------------------------------------------------ kernels
__global__ void k_rnvp_cond(const float* __restrict__ x, const float* __restrict__ m, int64_t n, int d,
                            float* __restrict__ cond) {
  const int64_t tot = n * d;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x)
    cond[i] = x[i] * m[i % d];
}

// one warp per row; y may alias x. first: ld = sum, else ld += sum. With m_next
// also cond_next = y * m_next, the next layer's conditioner input
__global__ void k_rnvp_couple(const float* x, const float* __restrict__ sraw, const float* __restrict__ tt,
                              const float* __restrict__ m, int64_t n, int d, float dt, int inverse, float* y,
                              float* __restrict__ ld, int first, const float* __restrict__ m_next,
                              float* __restrict__ cond_next) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
    float acc = 0.f;
    for (int j = lane; j < d; j += 32) {
      const int64_t e = r * d + j;
      const float mj = m[j], xv = x[e];
      const float s = tanhf(sraw[e]) * dt;        // MLPAffine: tanh(scale_MLP(c)) * dt
      const float t = tt[e] * dt;                 //            shift_MLP(c) * dt
      const float ya = inverse ? xv * expf(-s) - t : (xv + t) * expf(s);
      const float yv = (1.f - mj) * ya + mj * xv; // MaskedCouplingLayer mix
      y[e] = yv;
      if (m_next != nullptr) cond_next[e] = yv * m_next[j];
      acc += (1.f - mj) * s;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const float v = inverse ? -acc : acc;
      ld[r] = first ? v : ld[r] + v;
    }
  }
}

// adjoint of one forward coupling: gy (dL/dy) and gld (dL/d log-det, the
// same for every row) -> gx (the direct part; the conditioner's part is
// added later), and in place sraw -> dL/d sraw, tt -> dL/d tt
__global__ void k_rnvp_couple_bwd(const float* __restrict__ x, float* __restrict__ sraw, float* __restrict__ tt,
                                  const float* __restrict__ m, const float* __restrict__ gy, int64_t n, int d,
                                  float dt, float gld, float* __restrict__ gx) {
  const int64_t tot = n * d;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const float mj = m[e % d], xv = x[e];
    const float th = tanhf(sraw[e]);
    const float s = th * dt, t = tt[e] * dt;
    const float ex = expf(s);
    const float ya = (xv + t) * ex;
    const float g = gy[e];
    const float dya = (1.f - mj) * g;
    gx[e] = mj * g + dya * ex;
    const float ds = dya * ya + gld * (1.f - mj);
    sraw[e] = ds * dt * (1.f - th * th);
    tt[e] = dya * ex * dt;
  }
}

// per layer W2s^T, W2t^T [H, d] and W1^T [d, 2H]: the K-major operands of the
// backward GEMMs
__global__ void k_rnvp_transpose(const float* __restrict__ theta, RnvpGeom g, float* __restrict__ out) {
  const int64_t hd = (int64_t)g.H * g.d, per = 4 * hd;
  const float* th = theta + blockIdx.y * g.per_layer;
  float* o = out + blockIdx.y * per;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < per; e += (int64_t)gridDim.x * blockDim.x) {
    if (e < 2 * hd) {
      const int64_t q = e % hd, h = q / g.d, j = q % g.d;
      o[e] = th[(e < hd ? g.off_W2s : g.off_W2t) + j * g.H + h];
    } else {
      const int64_t q = e - 2 * hd, j = q / (2 * g.H), h = q % (2 * g.H);
      o[e] = th[h * g.d + j];
    }
  }
}

// column sums of dz [n, 2H], d sraw and d t [n, d] of layer blockIdx.z / 3 over
// row block blockIdx.y into part[parameter][row block]
__device__ __forceinline__ int rnvp_bias(const RnvpGeom& g, int which, int64_t& off) {
  off = which == 0 ? g.off_b1 : which == 1 ? g.off_b2s : g.off_b2t;
  return which == 0 ? 2 * g.H : g.d;
}
__global__ void k_rnvp_bias_partial(RnvpGeom g, const float* __restrict__ dz, const float* __restrict__ ds,
                                    const float* __restrict__ dt, int64_t n, int64_t rows_per, float* __restrict__ part) {
  const int l = blockIdx.z / 3, which = blockIdx.z % 3;
  int64_t off;
  const int cols = rnvp_bias(g, which, off), c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const float* src = (which == 0 ? dz : which == 1 ? ds : dt) + (int64_t)l * n * cols + c;
  const int64_t r0 = blockIdx.y * rows_per, r1 = r0 + rows_per < n ? r0 + rows_per : n;
  float v = 0.f;
#pragma unroll 16
  for (int64_t r = r0; r < r1; ++r) v += src[r * cols];
  const int64_t first = which == 0 ? 0 : which == 1 ? 2 * g.H : 2 * g.H + g.d;
  part[((int64_t)l * (2 * g.H + 2 * g.d) + first + c) * gridDim.y + blockIdx.y] = v;
}
__global__ void k_rnvp_bias_final(RnvpGeom g, const float* __restrict__ part, int rb, float* __restrict__ grad) {
  const int l = blockIdx.z / 3, which = blockIdx.z % 3;
  int64_t off;
  const int cols = rnvp_bias(g, which, off), c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const int64_t first = which == 0 ? 0 : which == 1 ? 2 * g.H : 2 * g.H + g.d;
  const float* p = part + ((int64_t)l * (2 * g.H + 2 * g.d) + first + c) * rb;
  float v = 0.f;
  for (int b = 0; b < rb; ++b) v += p[b];
  grad[l * g.per_layer + off + c] = v;
}
__global__ void k_rnvp_add(const float* __restrict__ part, int64_t n, float* __restrict__ grad) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    grad[e] += part[e];
}
// grad = sum of the slices (bias entries are overwritten by k_rnvp_bias_final)
__global__ void k_rnvp_sum_slices(const float* __restrict__ part, int S, int64_t n, float* __restrict__ grad) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    float v = 0.f;
#pragma unroll 4
    for (int z = 0; z < S; ++z) v += part[z * n + e];
    grad[e] = v;
  }
}

// log N(y; 0, I) + ld (realNVP.py:218-221: the standard normal, not the base distribution)
__global__ void k_rnvp_logprob(const float* __restrict__ y, const float* __restrict__ ld, int64_t n, int d,
                               float* __restrict__ logp) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
    float s = 0.f;
    for (int j = lane; j < d; j += 32) {
      const float v = y[r * d + j];
      s += v * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) logp[r] = ld[r] + (-0.5f * s - 0.5f * (float)d * logf(6.283185307179586f));
  }
}

// loss = -mean(logp) in fixed order (one block); gy = y / n seeds the backward
__global__ void k_rnvp_loss(const float* __restrict__ logp, int64_t n, float* __restrict__ loss) {
  __shared__ float sh[32];
  float s = 0.f;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += logp[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) *loss = -v / (float)n;
  }
}

__global__ void k_rnvp_scale(const float* __restrict__ y, int64_t tot, float c, float* __restrict__ out) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x)
    out[e] = y[e] * c;
}

// ------------------------------------------------------------------ layer passes
struct RnvpScratch {
  float* cond;   // [rows, d]
  float* h;      // [rows, 2H]
  float* sraw;   // [rows, d]
  float* tt;     // [rows, d]
};

static const float* layer_mask(const RnvpGeom& g, const float* aux, int l) { return aux + 2 * g.d + 2 + (int64_t)l * g.d; }

// the layer's conditioner on cond = x * m: h = relu(cond W1^T + b1), sraw, tt
static int rnvp_conditioner(cudaStream_t st, const RnvpGeom& g, const float* th, int64_t rows, const RnvpScratch& s) {
  const int d = g.d, H = g.H;
  G32Args a{};
  a.M = rows;
  a.p[0] = G32Problem{s.cond, th, th + g.off_b1, nullptr, s.h};
  a.lda = a.ldb = d;
  a.ldc = 2 * H;
  a.N = 2 * H;
  a.K = d;
  int rc = gemm_f32<G32_BIAS_RELU>(st, a, 1);
  if (rc) return rc;
  a.p[0] = G32Problem{s.h, th + g.off_W2s, th + g.off_b2s, nullptr, s.sraw};
  a.p[1] = G32Problem{s.h + H, th + g.off_W2t, th + g.off_b2t, nullptr, s.tt};
  a.lda = 2 * H;
  a.ldb = H;
  a.ldc = d;
  a.N = d;
  a.K = H;
  return gemm_f32<G32_BIAS>(st, a, 2);
}

// all layers, in place on x [rows, d] (forward: 0..L-1, inverse: L-1..0); ld = the summed log-det
static int rnvp_pass(cudaStream_t st, const RnvpGeom& g, const FmcRealNVP* f, float* x, int64_t rows, float* ld,
                     bool inverse, const RnvpScratch& s) {
  k_rnvp_cond<<<grid_for(rows * g.d), 256, 0, st>>>(x, layer_mask(g, f->aux, inverse ? g.L - 1 : 0), rows, g.d, s.cond);
  FMC_LAUNCH_CHECK();
  for (int i = 0; i < g.L; ++i) {
    const int l = inverse ? g.L - 1 - i : i;
    int rc = rnvp_conditioner(st, g, f->theta + (int64_t)l * g.per_layer, rows, s);
    if (rc) return rc;
    const float* next = i + 1 < g.L ? layer_mask(g, f->aux, inverse ? l - 1 : l + 1) : nullptr;
    k_rnvp_couple<<<warp_grid(rows), 256, 0, st>>>(x, s.sraw, s.tt, layer_mask(g, f->aux, l), rows, g.d, g.dt,
                                                   inverse ? 1 : 0, x, ld, i == 0 ? 1 : 0, next, s.cond);
    FMC_LAUNCH_CHECK();
  }
  return FMC_OK;
}

static size_t infer_floats(const RnvpGeom& g, int64_t rows) {
  return (size_t)rows * (4 * (size_t)g.d + 2 * (size_t)g.H) + (size_t)rows + 64 * 8;
}

static int carve_infer(const RnvpGeom& g, int64_t rows, void* ws, size_t ws_bytes, RnvpScratch& s, float** xa,
                       float** ld) {
  FMC_CHECK_ARG(ws != nullptr && ws_bytes >= infer_floats(g, rows) * sizeof(float),
                "workspace of %zu bytes is smaller than fmc_rnvp_workspace_size", ws_bytes);
  float* p = (float*)ws;
  auto take = [&](int64_t floats) {
    float* r = p;
    p += (floats + 63) / 64 * 64;   // 256-byte pieces: 16-byte copies where the shapes allow them
    return r;
  };
  s.cond = take(rows * g.d);
  s.h = take(rows * 2 * (int64_t)g.H);
  s.sraw = take(rows * g.d);
  s.tt = take(rows * g.d);
  *xa = take(rows * g.d);
  *ld = p;
  return FMC_OK;
}

// row slices of the weight gradients: enough 256 x 32 tiles for two CTAs per SM,
// at least 256 rows each (*most: a bound that only grows with n)
static int wgrad_slices(const RnvpGeom& g, int64_t n, int64_t* rows_per, int64_t* most = nullptr) {
  auto tiles = [](int64_t M, int64_t N) { return ((M + kK32M - 1) / kK32M) * ((N + kK32N - 1) / kK32N); };
  const int64_t per = g.L * (tiles(2 * g.H, g.d) + 2 * tiles(g.H, g.d));
  int64_t S = (4 * (int64_t)sm_count() + per - 1) / per;
  const int64_t by_rows = (n + 255) / 256;
  if (S > by_rows) S = by_rows;
  if (S > kMaxSlices) S = kMaxSlices;
  if (S < 1) S = 1;
  if (most) *most = S;
  *rows_per = ((n + S - 1) / S + kG32BK - 1) / kG32BK * kG32BK;
  return (int)((n + *rows_per - 1) / *rows_per);
}

static int bias_blocks(int64_t n) {
  const int64_t b = (n + 511) / 512;
  return (int)(b < 1 ? 1 : b > 128 ? 128 : b);
}

// Rows of a training chunk. A row keeps every layer's input, masked input, hidden
// activations, conditioner outputs (later their gradients) and hidden gradients,
// and two input gradients: 37 KB for 32 dims, 8 layers, H = 256. A batch runs in
// chunks of as many rows as kRnvpKeepBytes hold (461,000 there), their gradients
// added in order, so that the workspace grows by four bytes a row from there on: a
// million rows took 34.7 GiB without the chunks and take 16 with them.
constexpr size_t kRnvpKeepBytes = (size_t)16 << 30;
static size_t keep_floats_per_row(const RnvpGeom& g) {
  const size_t d = g.d, H = g.H, L = g.L;
  return (L + 1) * d + L * (3 * d + 4 * H) + 2 * d + 1;
}
static int64_t train_chunk(const RnvpGeom& g, int64_t n) {
  const int64_t most = (int64_t)(kRnvpKeepBytes / (4 * keep_floats_per_row(g))) / 256 * 256;
  const int64_t rows = most < 256 ? 256 : most;
  return n < rows ? n : rows;
}

static size_t train_floats(const RnvpGeom& g, int64_t n) {
  const size_t d = g.d, H = g.H, L = g.L;
  const int64_t m = train_chunk(g, n);
  int64_t rp, most;
  wgrad_slices(g, m, &rp, &most);
  return (size_t)m * keep_floats_per_row(g) + (size_t)n + (size_t)(most + 1) * g.n_params + L * 4 * H * d +
         L * (2 * H + 2 * d) * bias_blocks(m) + 64 * 14;
}

}  // namespace fmc

using namespace fmc;

extern "C" int fmc_rnvp_layout(const FmcRealNVP* flow, int64_t* n_params, int64_t* n_aux) {
  RnvpGeom g;
  int rc = rnvp_geom(flow, g);
  if (rc) return rc;
  if (n_params) *n_params = g.n_params;
  if (n_aux) *n_aux = g.n_aux;
  return FMC_OK;
}

extern "C" int fmc_rnvp_workspace_size(const FmcRealNVP* flow, int64_t n, int32_t mode, size_t* bytes) {
  RnvpGeom g;
  int rc = rnvp_geom(flow, g);
  if (rc) return rc;
  FMC_CHECK_ARG(bytes != nullptr && n >= 0, "bad arguments");
  const int64_t rows = n < kRnvpChunk ? (n > 0 ? n : 1) : kRnvpChunk;
  *bytes = (mode == 1 ? train_floats(g, n > 0 ? n : 1) : infer_floats(g, rows)) * sizeof(float);
  return FMC_OK;
}

static int rnvp_transform(const FmcRealNVP* flow, const float* in, int64_t n, float* out, float* logdet, void* ws,
                          size_t ws_bytes, void* stream, bool inverse) {
  RnvpGeom g;
  int rc = rnvp_geom(flow, g);
  if (rc) return rc;
  FMC_CHECK_ARG(n >= 0, "n < 0");
  if (n == 0) return FMC_OK;
  FMC_CHECK_ARG(in && out && logdet && flow->theta && flow->aux, "NULL array argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows = n < kRnvpChunk ? n : kRnvpChunk;
  RnvpScratch s;
  float *xa, *ldw;
  rc = carve_infer(g, rows, ws, ws_bytes, s, &xa, &ldw);
  if (rc) return rc;
  if (out != in) FMC_CUDA_TRY(cudaMemcpyAsync(out, in, sizeof(float) * n * g.d, cudaMemcpyDeviceToDevice, st));
  for (int64_t r0 = 0; r0 < n; r0 += rows) {
    const int64_t m = (n - r0 < rows) ? n - r0 : rows;
    rc = rnvp_pass(st, g, flow, out + r0 * g.d, m, logdet + r0, inverse, s);
    if (rc) return rc;
  }
  return FMC_OK;
}

extern "C" int fmc_rnvp_forward(const FmcRealNVP* flow, const float* x, int64_t n, float* y, float* logdet, void* ws,
                                size_t ws_bytes, void* stream) {
  return rnvp_transform(flow, x, n, y, logdet, ws, ws_bytes, stream, false);
}

extern "C" int fmc_rnvp_inverse(const FmcRealNVP* flow, const float* y, int64_t n, float* x, float* logdet, void* ws,
                                size_t ws_bytes, void* stream) {
  return rnvp_transform(flow, y, n, x, logdet, ws, ws_bytes, stream, true);
}

extern "C" int fmc_rnvp_log_prob(const FmcRealNVP* flow, const float* x, int64_t n, float* logp, void* ws,
                                 size_t ws_bytes, void* stream) {
  RnvpGeom g;
  int rc = rnvp_geom(flow, g);
  if (rc) return rc;
  FMC_CHECK_ARG(n >= 0, "n < 0");
  if (n == 0) return FMC_OK;
  FMC_CHECK_ARG(x && logp && flow->theta && flow->aux, "NULL array argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows = n < kRnvpChunk ? n : kRnvpChunk;
  RnvpScratch s;
  float *xa, *ld;
  rc = carve_infer(g, rows, ws, ws_bytes, s, &xa, &ld);
  if (rc) return rc;
  for (int64_t r0 = 0; r0 < n; r0 += rows) {
    const int64_t m = (n - r0 < rows) ? n - r0 : rows;
    k_standardize<<<grid_for(m * g.d), 256, 0, st>>>(x + r0 * g.d, m, g.d, flow->aux, xa);
    FMC_LAUNCH_CHECK();
    rc = rnvp_pass(st, g, flow, xa, m, ld, false, s);
    if (rc) return rc;
    k_rnvp_logprob<<<warp_grid(m), 256, 0, st>>>(xa, ld, m, g.d, logp + r0);
    FMC_LAUNCH_CHECK();
  }
  return FMC_OK;
}

extern "C" int fmc_rnvp_sample(const FmcRealNVP* flow, uint64_t seed, uint64_t counter, const float* z, int64_t n,
                               float* out, void* ws, size_t ws_bytes, void* stream) {
  RnvpGeom g;
  int rc = rnvp_geom(flow, g);
  if (rc) return rc;
  FMC_CHECK_ARG(n >= 0, "n < 0");
  if (n == 0) return FMC_OK;
  FMC_CHECK_ARG(out && flow->theta && flow->aux, "NULL array argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows = n < kRnvpChunk ? n : kRnvpChunk;
  RnvpScratch s;
  float *xa, *ld;
  rc = carve_infer(g, rows, ws, ws_bytes, s, &xa, &ld);
  if (rc) return rc;
  // base_dist.sample: sqrt(c) z for the Gaussian(0, c I) base (common.py:288-293)
  const Rng rng{(uint32_t)seed, (uint32_t)(seed >> 32), counter, rng_epoch()};
  k_base_sample<<<grid_for(n * g.d), 256, 0, st>>>(z, rng, n, g.d, flow->aux, out);
  FMC_LAUNCH_CHECK();
  for (int64_t r0 = 0; r0 < n; r0 += rows) {
    const int64_t m = (n - r0 < rows) ? n - r0 : rows;
    rc = rnvp_pass(st, g, flow, out + r0 * g.d, m, ld, true, s);
    if (rc) return rc;
  }
  k_destandardize<<<grid_for(n * g.d), 256, 0, st>>>(out, n, g.d, flow->aux);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}

extern "C" int fmc_rnvp_loss_grad(const FmcRealNVP* flow, const float* x, int64_t n, float* loss, float* grad,
                                  void* ws, size_t ws_bytes, void* stream) {
  RnvpGeom g;
  int rc = rnvp_geom(flow, g);
  if (rc) return rc;
  FMC_CHECK_ARG(n >= 1, "n=%lld < 1", (long long)n);
  FMC_CHECK_ARG(x && loss && grad && flow->theta && flow->aux, "NULL array argument");
  FMC_CHECK_ARG(ws != nullptr && ws_bytes >= train_floats(g, n) * sizeof(float),
                "workspace of %zu bytes is smaller than fmc_rnvp_workspace_size", ws_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  const int d = g.d, H = g.H;
  const int64_t chunk = train_chunk(g, n);
  const int64_t cd = chunk * d, ch = chunk * 2 * (int64_t)H;
  float* p = (float*)ws;
  auto take = [&](int64_t floats) {
    float* r = p;
    p += (floats + 63) / 64 * 64;   // 256-byte pieces: 16-byte copies where the shapes allow them
    return r;
  };
  float* X = take((g.L + 1) * cd);   // layer inputs, X[L] = y
  float* cond = take(g.L * cd);
  float* sraw = take(g.L * cd);
  float* tt = take(g.L * cd);
  float* h = take(g.L * ch);
  float* dz = take(g.L * ch);
  float* gin[2] = {take(cd), take(cd)};
  float* ld = take(chunk);
  float* logp = take(n);
  float* wt = take((int64_t)g.L * 4 * H * d);
  float* bpart = take((int64_t)g.L * (2 * H + 2 * d) * bias_blocks(chunk));
  float* cgrad = take(g.n_params);   // a later chunk's gradient
  float* part = p;
  k_rnvp_transpose<<<dim3((unsigned)grid_for(4ll * H * d, 1), (unsigned)g.L), 256, 0, st>>>(flow->theta, g, wt);
  FMC_LAUNCH_CHECK();
  const float gld = -1.f / (float)n;
  constexpr int ksmem = kG32Stages * kK32StageFloats * 4;
  FMC_CUDA_TRY(cudaFuncSetAttribute(k_kouter_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, ksmem));

  for (int64_t r0 = 0; r0 < n; r0 += chunk) {
    const int64_t m = n - r0 < chunk ? n - r0 : chunk;
    const int64_t nd = m * d, nh = m * 2 * (int64_t)H;
    // forward, keeping every layer's activations
    k_standardize<<<grid_for(nd), 256, 0, st>>>(x + r0 * d, m, d, flow->aux, X);
    FMC_LAUNCH_CHECK();
    k_rnvp_cond<<<grid_for(nd), 256, 0, st>>>(X, layer_mask(g, flow->aux, 0), m, d, cond);
    FMC_LAUNCH_CHECK();
    for (int l = 0; l < g.L; ++l) {
      const RnvpScratch s{cond + l * nd, h + l * nh, sraw + l * nd, tt + l * nd};
      rc = rnvp_conditioner(st, g, flow->theta + (int64_t)l * g.per_layer, m, s);
      if (rc) return rc;
      const bool last = l + 1 == g.L;
      k_rnvp_couple<<<warp_grid(m), 256, 0, st>>>(X + l * nd, s.sraw, s.tt, layer_mask(g, flow->aux, l), m, d, g.dt, 0,
                                                  X + (l + 1) * nd, ld, l == 0 ? 1 : 0,
                                                  last ? nullptr : layer_mask(g, flow->aux, l + 1),
                                                  last ? nullptr : cond + (l + 1) * nd);
      FMC_LAUNCH_CHECK();
    }
    float* y = X + (int64_t)g.L * nd;
    k_rnvp_logprob<<<warp_grid(m), 256, 0, st>>>(y, ld, m, d, logp + r0);
    FMC_LAUNCH_CHECK();

    // backward: loss = -mean(ld + log N(y)) -> dL/dy = y / n, dL/d ld = -1 / n
    float *gy = gin[0], *gx = gin[1];
    k_rnvp_scale<<<grid_for(nd), 256, 0, st>>>(y, nd, 1.f / (float)n, gy);
    FMC_LAUNCH_CHECK();
    for (int l = g.L - 1; l >= 0; --l) {
      const float* mk = layer_mask(g, flow->aux, l);
      const float* wl = wt + (int64_t)l * 4 * H * d;
      k_rnvp_couple_bwd<<<grid_for(nd), 256, 0, st>>>(X + l * nd, sraw + l * nd, tt + l * nd, mk, gy, m, d, g.dt, gld,
                                                      gx);
      FMC_LAUNCH_CHECK();
      // dz = [dsraw W2s, dtt W2t] masked by relu'
      G32Args a{};
      a.M = m;
      a.p[0] = G32Problem{sraw + l * nd, wl, nullptr, h + l * nh, dz + l * nh};
      a.p[1] = G32Problem{tt + l * nd, wl + (int64_t)H * d, nullptr, h + l * nh + H, dz + l * nh + H};
      a.lda = a.ldb = d;
      a.ldaux = a.ldc = 2 * H;
      a.N = H;
      a.K = d;
      rc = gemm_f32<G32_DRELU>(st, a, 2);
      if (rc) return rc;
      // gx += (dz W1) * mask
      a.p[0] = G32Problem{dz + l * nh, wl + 2ll * H * d, mk, nullptr, gx};
      a.lda = a.ldb = 2 * H;
      a.ldc = d;
      a.N = d;
      a.K = 2 * H;
      rc = gemm_f32<G32_ADD_MASKED>(st, a, 1);
      if (rc) return rc;
      float* t = gy;
      gy = gx;
      gx = t;
    }
    // weight and bias gradients of all layers over the chunk. The second
    // Linears' as h^T d(output), stored transposed: the wide side is the tall
    // operand of the 256 x 32 tiles
    float* out = r0 == 0 ? grad : cgrad;
    int64_t rows_per = 0;
    const int slices = wgrad_slices(g, m, &rows_per), rb = bias_blocks(m);
    K32Args k{};
    k.p[0] = K32Problem{dz, cond, nh, nd, 2 * H, d, 2 * H, d, 0, d, 1};
    k.p[1] = K32Problem{h, sraw, nh, nd, 2 * H, d, H, d, g.off_W2s, 1, H};
    k.p[2] = K32Problem{h + H, tt, nh, nd, 2 * H, d, H, d, g.off_W2t, 1, H};
    k.n_problems = 3;
    k.rows = m;
    k.rows_per_slice = rows_per;
    k.per_layer = g.per_layer;
    k.n_params = g.n_params;
    k.part = part;
    const unsigned tiles = (unsigned)(((2 * H + kK32M - 1) / kK32M) * ((d + kK32N - 1) / kK32N));
    k_kouter_f32<<<dim3(tiles, (unsigned)slices, (unsigned)(3 * g.L)), kK32Threads, ksmem, st>>>(k);
    FMC_LAUNCH_CHECK();
    k_rnvp_sum_slices<<<grid_for(g.n_params), 256, 0, st>>>(part, slices, g.n_params, out);
    FMC_LAUNCH_CHECK();
    const unsigned cb = (unsigned)((2 * H > d ? 2 * H : d) + 127) / 128;
    k_rnvp_bias_partial<<<dim3(cb, (unsigned)rb, (unsigned)(3 * g.L)), 128, 0, st>>>(g, dz, sraw, tt, m, (m + rb - 1) / rb,
                                                                                    bpart);
    FMC_LAUNCH_CHECK();
    k_rnvp_bias_final<<<dim3(cb, 1, (unsigned)(3 * g.L)), 128, 0, st>>>(g, bpart, rb, out);
    FMC_LAUNCH_CHECK();
    if (r0 > 0) {
      k_rnvp_add<<<grid_for(g.n_params), 256, 0, st>>>(cgrad, g.n_params, grad);
      FMC_LAUNCH_CHECK();
    }
  }
  k_rnvp_loss<<<1, 1024, 0, st>>>(logp, n, loss);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}
