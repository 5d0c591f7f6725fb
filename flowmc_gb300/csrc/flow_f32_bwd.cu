// flow_f32_bwd.cu -- gradient of the FP32 flow loss in seven launches, from the
// layer inputs and activations the fused forward pass (flow_f32.cu) left behind
// (NFModel.loss_fn's reverse pass, nf_model/base.py:98-125).
//
//   k_flow_f32_bwd   a tile of rows through every layer in reverse: spline
//                    adjoint, conditioner input gradients, ScalarAffine adjoint.
//                    Leaves the gradients of every Linear's outputs and of every
//                    layer's affine output.
//   k_wgrad_f32      all weight gradients as one grid of 128 x 64 tiles over
//                    (layer, Linear, outputs, inputs, slice of the rows), then
//   k_sum_wgrad      the sum of the slices
//   k_bias_partial, k_bias_final    all bias gradients
//   k_affine_layers, k_affine_final the affine parameters' gradients
//
// Before, every layer took about 25 launches: the conditioner recomputed into
// HBM, a spline adjoint whose lanes strode 3K + 1 floats, three 64 x 64-tile
// input-gradient GEMMs, three split-K weight gradients, three column-sum pairs.
// Activations are now kept instead of recomputed (per row and layer n_c + sum H +
// n_t (3K + 1) floats), in tiles of [column][R rows]; output gradients are
// row-major. Every sum over the batch keeps the order of the launches it
// replaces (row slices, row blocks, warps), so the gradients are the same bits:
// a training trajectory crosses spline knots, and gradients that differ in the
// last place part from each other there after an optimiser step.
//
// Bound by FMA issue and, with eight warps per SM, by the latency of the spline
// adjoint. Measured on GB300, loss + gradient + AdamW: 16,384 rows of the 32-D
// flow (8 x [128, 128] x 10 bins) 5.88 -> 2.38 ms (forward 0.79, backward 0.97,
// weight gradients 0.44 = 48 TFLOP/s, biases 0.07); 10,000 rows of the 5-D flow
// (4 x [32, 32] x 8 bins) 1.02 -> 0.34 ms.
#include <algorithm>
#include "flow_f32.cuh"
#include "flow_f32.h"
#include "gemm_simt.cuh"
#include "train_sums.cuh"

namespace fmc {

struct FlowBwdArgs {
  FlowShape s;
  const float* theta;
  const float* aux;
  const float* save;   // [L + 1, n, d]
  const float* acts;   // saved activations
  float* gout;         // output gradients [Linear of a layer][rows][round_up(out, 4)]
  float* gaff;         // [L, n, d]: dL/d (affine output)
  int64_t n, tiles;
  float inv_n;
  int ldx, act_floats;
};

// shared memory (floats): xs, gy [R][ldx] (the layer's affine output and dL/d
// of it), two tiles of act_floats ([column][R + 4]), weight stages
template <int K, int R>
__global__ void __launch_bounds__(FlowTile<R>::NT, 2) k_flow_f32_bwd(const __grid_constant__ FlowBwdArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int P = 3 * K + 1;
  using T = FlowTile<R>;
  using U = FlowTileT<R>;
  constexpr int NT = T::NT, NW = NT / 32;
  const FlowShape& s = a.s;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int d = s.d;
  float* xs = sm;
  float* gy = xs + R * a.ldx;
  float* t0 = gy + R * a.ldx;
  float* t1 = t0 + a.act_floats;
  float* ring = t1 + a.act_floats;
  const int r0 = (wid / T::WC) * 32 + flow_lane_row();
  const int64_t row_base = (int64_t)blockIdx.x * R;
  const int rows = (int)(a.n - row_base < R ? a.n - row_base : R);

  WtStream<NT, T::ST> w;
  w.begin(&s, a.theta, ring);
  int slot = 0;

  // dL/dy = y / (c n) at the flow's output; rows past n carry no gradient
  {
    const float c = a.aux[2 * d];
    for (int r = wid; r < R; r += NW)
      for (int j = lane; j < d; j += 32)
        gy[r * a.ldx + j] = r < rows ? a.save[((int64_t)s.L * a.n + row_base + r) * d + j] / c * a.inv_n : 0.f;
  }
  const int row = tid % R;
  const float gld = row < rows ? -a.inv_n : 0.f;

  for (int l = s.L - 1; l >= 0; --l) {
    const float* th = a.theta + s.layer_off(l);
    const int nc = s.nc(l), nt = s.nt(l), cpar = s.cpar(l), tpar = s.tpar(l);
    const float sc = __ldg(th), sh = __ldg(th + 1), es = expf(sc);
    for (int r = wid; r < R; r += NW)
      for (int j = lane; j < d; j += 32)
        xs[r * a.ldx + j] =
            r < rows ? scalar_affine(a.save[((int64_t)l * a.n + row_base + r) * d + j], es, sh, 0) : 0.f;

    uint64_t acc[T::TQ][T::TN][2];
#pragma unroll
    for (int q = 0; q < T::TQ; ++q)
#pragma unroll
      for (int j = 0; j < T::TN; ++j) acc[q][j][0] = acc[q][j][1] = 0ull;

    // ---- splines and the last Linear's input gradient, a group of coordinates at a time
    const int out = nt * P, tc = s.dg * P, hin = s.in(l, s.nh);
    const float* raw = a.acts + ((s.act_base(l) + s.act_col(l, s.nh + 1)) * a.tiles + (int64_t)blockIdx.x * out) * R;
    const int gp = s.gpad(l, s.nh);
    float* graw = a.gout + s.gcol(l, s.nh) * (a.tiles * R) + row_base * gp;
    // raw tiles by cp.async, the next group's while this one is worked on; the
    // copies ride in the weight stream's groups
    auto fetch = [&](int n0, float* tile) {
      const int N = min(tc, out - n0), Np = (N + 15) & ~15;
      const float* src = raw + (int64_t)n0 * R;
      for (int e = tid; e < Np * (R / 4); e += NT) {
        const int c = e / (R / 4), r = (e % (R / 4)) * 4;
        float* dst = tile + c * T::LD + r;
        if (c < N)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                       "l"(src + c * R + r));
        else
          *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    float* tile = t0;
    float* next = t1;
    fetch(0, tile);
    for (int n0 = 0, c0t = 0; n0 < out; n0 += tc, c0t += s.dg) {
      const int N = min(tc, out - n0);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();   // the tile, xs and gy are complete, the other tile is free
      if (n0 + tc < out) fetch(n0 + tc, next);
      const int items = (N / P) * R;
      for (int e = tid; e < items; e += NT) {
        const int t = e / R;
        float prm[P];
        float* tp = tile + t * P * T::LD + row;
#pragma unroll
        for (int p = 0; p < P; ++p) prm[p] = tp[p * T::LD];
        const int j = row * a.ldx + 2 * (c0t + t) + tpar;
        gy[j] = rqs_adjoint<K>(prm, xs[j], s.cfg, gy[j], gld, [&](int p, float v) { tp[p * T::LD] = v; });
      }
      __syncthreads();
      // rows of d raw: eight columns x four rows per warp access (distinct banks,
      // whole sectors)
      for (int e = wid; e < (N + 7) / 8 * (R / 4); e += NW) {
        const int c = e / (R / 4) * 8 + (lane & 7), r = e % (R / 4) * 4 + (lane >> 3);
        if (c < N) graw[(int64_t)r * gp + n0 + c] = tile[c * T::LD + r];
      }
      flow_product_t<R>(w, ring, slot, tile, hin, N, r0, acc);
      float* t = tile;
      tile = next;
      next = t;
    }

    // ---- hidden Linears: dz = (gradient) (1 - h^2), then through the Linear
    float* cur = tile;   // not the last group's
    float* other = next;
    for (int i = s.nh - 1; i >= 0; --i) {
      const int H = s.out(l, i), Hp = (H + 15) & ~15;
      const float* h = a.acts + ((s.act_base(l) + s.act_col(l, i + 1)) * a.tiles + (int64_t)blockIdx.x * H) * R;
      const int zp = s.gpad(l, i);
      float* dz = a.gout + s.gcol(l, i) * (a.tiles * R) + row_base * zp;
      if (i < s.nh - 1) __syncthreads();   // `cur` was read by the product before the last
#pragma unroll
      for (int g = 0; g < U::NG; ++g) {
        const int c0 = U::col0() + 8 * U::E * g;
#pragma unroll
        for (int q = 0; q < T::TQ; ++q) {
          float v[U::E][4];
#pragma unroll
          for (int e = 0; e < U::E; ++e) {
            const int c = c0 + e, j = U::E * g + e;
            f2_unpack(acc[q][j][0], v[e][0], v[e][1]);
            f2_unpack(acc[q][j][1], v[e][2], v[e][3]);
            acc[q][j][0] = acc[q][j][1] = 0ull;
            float4 hv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c < H) hv = *reinterpret_cast<const float4*>(h + (int64_t)c * R + r0 + 16 * q);
            v[e][0] = c < H ? v[e][0] * (1.f - hv.x * hv.x) : 0.f;
            v[e][1] = c < H ? v[e][1] * (1.f - hv.y * hv.y) : 0.f;
            v[e][2] = c < H ? v[e][2] * (1.f - hv.z * hv.z) : 0.f;
            v[e][3] = c < H ? v[e][3] * (1.f - hv.w * hv.w) : 0.f;
            if (c < Hp)
              *reinterpret_cast<float4*>(cur + c * T::LD + r0 + 16 * q) =
                  make_float4(v[e][0], v[e][1], v[e][2], v[e][3]);
          }
          if (c0 < zp) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              float* o = dz + (int64_t)(r0 + 16 * q + r) * zp + c0;
              if constexpr (U::E == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0][r], v[1][r], v[2][r], v[3][r]);
              else *reinterpret_cast<float2*>(o) = make_float2(v[0][r], v[1][r]);
            }
          }
        }
      }
      flow_product_t<R>(w, ring, slot, cur, s.in(l, i), H, r0, acc);
      float* t = cur;
      cur = other;
      other = t;
    }
    // ---- the conditioning coordinates' gradient, ScalarAffine adjoint
#pragma unroll
    for (int j = 0; j < T::TN; ++j) {
      const int c = U::col0() + 8 * U::E * (j / U::E) + j % U::E;
      if (c < nc) {
#pragma unroll
        for (int q = 0; q < T::TQ; ++q) {
          float4 v;
          f2_unpack(acc[q][j][0], v.x, v.y);
          f2_unpack(acc[q][j][1], v.z, v.w);
          float* g = gy + (r0 + 16 * q) * a.ldx + 2 * c + cpar;
          g[0] += v.x;
          g[a.ldx] += v.y;
          g[2 * a.ldx] += v.z;
          g[3 * a.ldx] += v.w;
        }
      }
    }
    __syncthreads();
    for (int r = wid; r < R; r += NW)
      for (int j = lane; j < d; j += 32) {
        const float g = gy[r * a.ldx + j];
        if (r < rows) a.gaff[((int64_t)l * a.n + row_base + r) * d + j] = g;
        gy[r * a.ldx + j] = g * es;
      }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ weight gradients
constexpr int kMaxLin = FMC_MAX_HIDDEN + 1;

// row slices of the weight gradients of Linear i of an even / odd layer
struct WgradSlices {
  int count[2][kMaxLin];
  int64_t rows[2][kMaxLin];
  int64_t part_off[2][kMaxLin];   // floats before this Linear's partials within a layer
  int64_t part_layer[2];          // floats of a layer's partials
  __host__ __device__ int64_t part(int l, int i) const {
    return (int64_t)(l / 2) * (part_layer[0] + part_layer[1]) + (l & 1) * part_layer[0] + part_off[l & 1][i];
  }
};

struct WgradArgs {
  FlowShape s;
  WgradSlices z;
  const float* acts;
  const float* gout;
  float* part;          // [layer][Linear][slice][out, in]
  int64_t n, tiles;
  int per_pair;         // tile items of an even and an odd layer together
};

constexpr int kWgM = 128, kWgN = 64, kWgThreads = 128, kWgStages = 4;
constexpr int kWgStageFloats = kFlowBK * kWgM + kWgN * kFlowPitch;

__host__ __device__ inline int wg_items(const FlowShape& s, int l, int i) {
  return ((s.out(l, i) + kWgM - 1) / kWgM) * ((s.in(l, i) + kWgN - 1) / kWgN);
}

// part[slice][m][n] = sum over the slice's rows of G[row][m] X[n][row], one FMA
// chain per element in row order. Packed FMAs over two adjacent m (G rows are
// m-contiguous), X's value in both halves; 16 x 4 outputs per thread, four warps
// of 64 x 32, 16 rows per stage, three stages in flight. FMA-bound.
template <int R>
__global__ void __launch_bounds__(kWgThreads, 2) k_wgrad_f32(const __grid_constant__ WgradArgs a) {
  extern __shared__ __align__(16) float sm[];
  const FlowShape& s = a.s;
  // item -> (layer, Linear, m tile, n tile)
  int it = blockIdx.x, l = it / a.per_pair * 2;
  it %= a.per_pair;
  int i = 0;
  for (;;) {
    const int n = wg_items(s, l, i);
    if (it < n) break;
    it -= n;
    if (++i > s.nh) {
      i = 0;
      ++l;
    }
  }
  // the absent odd layer of the last pair; slices this Linear does not have
  if (l >= s.L || (int)blockIdx.y >= a.z.count[l & 1][i]) return;
  const int M = s.out(l, i), N = s.in(l, i), tn = (N + kWgN - 1) / kWgN, gp = s.gpad(l, i);
  const int m0 = it / tn * kWgM, n0 = it % tn * kWgN;
  const float* G = a.gout + s.gcol(l, i) * (a.tiles * R) + m0;
  const float* X = a.acts + (s.act_base(l) + s.act_col(l, i)) * a.tiles * R;
  const int64_t k_begin = (int64_t)blockIdx.y * a.z.rows[l & 1][i];
  const int64_t k_end = k_begin + a.z.rows[l & 1][i] < a.n ? k_begin + a.z.rows[l & 1][i] : a.n;   // rows past n: zero G
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
  const int gr = tid >> 5, gc = (tid & 31) * 4;      // copies of G: rows gr + 4 q, 16 bytes at column gc
  const int xn = tid >> 2, xk = (tid & 3) * 4;       // of X: rows xn + 32 q, 16 bytes at row offset xk
  auto issue = [&](int64_t k, int slot) {
    if (k < k_end) {
      const uint32_t dst = sbase + slot * (4 * kWgStageFloats);
      if (m0 + gc < gp) {
        const float* g = G + (k + gr) * gp + gc;
#pragma unroll
        for (int q = 0; q < kFlowBK / 4; ++q)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4 * ((gr + 4 * q) * kWgM + gc)),
                       "l"(g + (int64_t)4 * q * gp));
      }
      const float* x = X + (k / R * N + n0 + xn) * R + (int)(k % R) + xk;
#pragma unroll
      for (int q = 0; q < kWgN / 32; ++q)
        if (n0 + xn + 32 * q < N)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                           dst + 4 * (kFlowBK * kWgM + (xn + 32 * q) * kFlowPitch + xk)),
                       "l"(x + (int64_t)32 * q * R));
    }
    asm volatile("cp.async.commit_group;");
  };
  const int mr = (wid >> 1) * 64 + (lane >> 3) * 4, nr = (wid & 1) * 32 + (lane & 7);   // outputs mr + 16 p + 0..3, nr + 8 q
  uint64_t acc[4][4][2];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q][0] = acc[p][q][1] = 0ull;
  const bool on = m0 + (wid >> 1) * 64 < M && n0 + (wid & 1) * 32 < N;
#pragma unroll
  for (int q = 0; q < kWgStages - 1; ++q) issue(k_begin + q * kFlowBK, q);
  int slot = 0;
  for (int64_t k = k_begin; k < k_end; k += kFlowBK) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kWgStages - 2) : "memory");
    __syncthreads();
    issue(k + (kWgStages - 1) * kFlowBK, slot == 0 ? kWgStages - 1 : slot - 1);
    if (on) {
      const float* As = sm + slot * kWgStageFloats + mr;
      const float* Bs = sm + slot * kWgStageFloats + kFlowBK * kWgM + nr * kFlowPitch;
#pragma unroll
      for (int kk = 0; kk < kFlowBK; kk += 4) {
        float4 b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = *reinterpret_cast<const float4*>(Bs + 8 * q * kFlowPitch + kk);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          uint64_t bb[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float v = r == 0 ? b[q].x : r == 1 ? b[q].y : r == 2 ? b[q].z : b[q].w;
            bb[q] = f2_pack(v, v);
          }
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(As + (kk + r) * kWgM + 16 * p);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              acc[p][q][0] = f2_fma(v.x, bb[q], acc[p][q][0]);
              acc[p][q][1] = f2_fma(v.y, bb[q], acc[p][q][1]);
            }
          }
        }
      }
    }
    slot = slot + 1 == kWgStages ? 0 : slot + 1;
  }
  float* out = a.part + a.z.part(l, i) + (int64_t)blockIdx.y * M * N;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int nn = n0 + nr + 8 * q, m = m0 + mr + 16 * p;
      float v[4];
      f2_unpack(acc[p][q][0], v[0], v[1]);
      f2_unpack(acc[p][q][1], v[2], v[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (m + e < M && nn < N) out[(int64_t)(m + e) * N + nn] = v[e];
    }
}

// weights of Linear blockIdx.y % (nh + 1) of layer blockIdx.y / (nh + 1): the sum of its slices
__global__ void k_sum_wgrad(const __grid_constant__ FlowShape s, const __grid_constant__ WgradSlices z,
                            const float* __restrict__ part, float* __restrict__ grad) {
  const int l = blockIdx.y / (s.nh + 1), i = blockIdx.y % (s.nh + 1);
  const int64_t base = s.layer_off(l) + s.w_off(l, i), cnt = (int64_t)s.out(l, i) * s.in(l, i);
  const float* p = part + z.part(l, i);
  const int S = z.count[l & 1][i];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x) {
    float v = 0.f;
#pragma unroll 4
    for (int q = 0; q < S; ++q) v += p[q * cnt + e];
    grad[base + e] = v;
  }
}

// column sums of every output gradient over row block blockIdx.y, rows in order
__global__ void k_bias_partial(const __grid_constant__ FlowShape s, const float* __restrict__ gout, int64_t n,
                               int64_t rows_pad, int64_t rows_per, float* __restrict__ part) {
  const int l = blockIdx.z / (s.nh + 1), i = blockIdx.z % (s.nh + 1);
  const int c = blockIdx.x * blockDim.x + threadIdx.x, gp = s.gpad(l, i);
  if (c >= s.out(l, i)) return;
  const int64_t col = s.gcol(l, i);
  const float* g = gout + col * rows_pad + c;
  const int64_t r0 = blockIdx.y * rows_per, r1 = r0 + rows_per < n ? r0 + rows_per : n;
  float v = 0.f;
#pragma unroll 32   // the adds are one chain, the loads are not
  for (int64_t r = r0; r < r1; ++r) v += g[r * gp];
  part[(col + c) * gridDim.y + blockIdx.y] = v;
}

__global__ void k_bias_final(const __grid_constant__ FlowShape s, const float* __restrict__ part, int rb,
                             float* __restrict__ grad) {
  const int l = blockIdx.z / (s.nh + 1), i = blockIdx.z % (s.nh + 1);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= s.out(l, i)) return;
  const float* p = part + (s.gcol(l, i) + c) * rb;
  float v = 0.f;
  for (int b = 0; b < rb; ++b) v += p[b];
  grad[s.layer_off(l) + s.w_off(l, i) + (int64_t)s.out(l, i) * s.in(l, i) + c] = v;
}

// the affine parameters' sums of layer blockIdx.y
__global__ void __launch_bounds__(256) k_affine_layers(const __grid_constant__ FlowShape s, const float* __restrict__ theta,
                                                       const float* __restrict__ save, const float* __restrict__ gaff,
                                                       int64_t n, float* __restrict__ part) {
  const int l = blockIdx.y, d = s.d;
  const float* th = theta + s.layer_off(l);
  const float sh = th[1], es = expf(th[0]);
  const float* xin = save + (int64_t)l * n * d;
  const float* ga = gaff + (int64_t)l * n * d;
  affine_sums(n, d, part + (int64_t)l * gridDim.x * 2, [&](int64_t r, int j, float& g, float& x, float& gv) {
    g = ga[r * d + j];
    x = scalar_affine(xin[r * d + j], es, sh, 0);
    gv = __fmul_rn(g, es);
  });
}

__global__ void k_affine_final(const __grid_constant__ FlowShape s, const float* __restrict__ part, int nb, float ld_term,
                               float* __restrict__ grad) {
  affine_param_grad(part + (int64_t)blockIdx.x * nb * 2, nb, ld_term, grad + s.layer_off(blockIdx.x));
}

// ------------------------------------------------------------------ host
static size_t bwd_smem(const FlowGeom& g, int R, FlowBwdArgs& a) {
  const FlowShape s = flow_shape(g);
  a.s = s;
  a.ldx = g.d | 1;
  int hm = (s.dg * s.P + 15) & ~15;
  for (int i = 0; i < g.nh; ++i) hm = ((g.H[i] + 15) & ~15) > hm ? ((g.H[i] + 15) & ~15) : hm;
  a.act_floats = hm * (R + 4);
  const int st = R >= 64 ? FlowTile<64>::ST : FlowTile<16>::ST;
  return sizeof(float) * (2 * (size_t)R * a.ldx + 2 * (size_t)a.act_floats + st * kFlowBK * kFlowCols);
}

// The fastest way to train on n rows, from estimates like flow_f32_route's
// (microseconds, both passes). What drives them:
//   S, T   stages of a layer's forward and backward products, G coordinate groups
//   t      row tiles on the fullest SM, f and b the rounds they run in forward and
//          backward (two CTAs share an SM where shared memory allows it)
// and the weight gradients' multiply-adds, which all ways have alike.
// Coefficients fitted to 750 random calls (GB300; 3 to 250 dims, 8 to 128 units, one
// to three hidden layers, 2 to 16 bins, 1 to 8 layers, 20 to 60,000 rows), which
// they reproduce within 15 % (16 and 64 rows) and 21 % (layers) for nine calls in
// ten. The way taken was on average 0.1 % and at worst 13 % behind the fastest of the
// three, and at worst 6 % behind the layers. 64 rows wherever they fill the SMs, 16
// otherwise, was 4 % behind on average and up to 1.7 times the layers' time:
// 250-D, 2 bins, one hidden layer of 48 units, 2 layers, 12,000 rows 952 us by
// layers, 1,616 in 64-row tiles, 851 in 16-row ones; 250-D, 16 bins, [48, 48], 4 layers,
// 1,000 rows 2,739 us by layers, 3,227 in 16-row tiles.
FlowGradRoute flow_f32_grad_route(const FlowGeom& g, int64_t n) {
  FlowGradRoute route{0, false};
  if (n < 1 || g.nc_max() > kFlowCols) return route;   // (a size may be asked for no rows)
  for (int i = 0; i < g.nh; ++i)
    if (g.H[i] > kFlowCols) return route;
  const FlowShape s = flow_shape(g);
  double S = 0, T = 0, G = 0, steps = 0, back = 0, macs = 0, raw = 0;   // means over the two layer parities
  for (int l = 0; l < 2; ++l)
    for (int i = 0; i <= g.nh; ++i) {
      const int in = s.in(l, i), out = s.out(l, i), tc = s.tile_cols(i);
      const int ks = (in + kFlowBK - 1) / kFlowBK;
      back += 0.5 * ((out + kFlowBK - 1) / kFlowBK);
      S += 0.5 * ((out + tc - 1) / tc) * ks;
      for (int n0 = 0; n0 < out; n0 += tc) T += 0.5 * ((std::min(tc, out - n0) + kFlowBK - 1) / kFlowBK);
      steps += 0.5 * ks;
      macs += 0.5e-6 * ((out + 63) / 64 * 64) * (ks * kFlowBK);
      if (i == g.nh) {
        G += 0.5 * ((out + tc - 1) / tc);
        raw += 0.5e-6 * out;
      }
    }
  const double L = g.L, nr = (double)n;
  // the launches per layer: chains of 16-deep steps forward and back, 32 splines a warp
  const double layers = 39.8 + L * (93.2 + 7.13 * steps + 0.402 * back + 0.705 * ((g.d + 63) / 64) * g.P +
                                    nr * (0.166 * macs + 15.9 * raw + 4.29e-3));
  double fused = 0.0;
  for (int R = 16; R <= 64; R += 48) {
    FlowBwdArgs a{};
    size_t fwd = 0;
    const size_t bwd = bwd_smem(g, R, a);
    if (bwd > 227 * 1024 || !flow_f32_tile_fits(g, R, &fwd)) continue;
    const double t = ceil(ceil((double)n / R) / sm_count());
    const double f = ceil(t / (2 * (fwd + 1024) <= 228 * 1024 ? 2 : 1));
    const double b = ceil(t / (2 * (bwd + 1024) <= 228 * 1024 ? 2 : 1));
    const double est =
        R == 16 ? 60.1 + L * (f * 0.213 * S + t * (0.481 * S + 0.144 * T + 0.0829 * g.d) +
                              b * (12.5 + 0.441 * T + 0.268 * G * g.K) + nr * 0.0375 * macs)
                : 78.9 + L * (f * (19.9 + 1.44 * G) + t * (0.896 * S + 0.157 * T + 0.53 * g.d) + b * 1.59 * T +
                              nr * (0.0609 * macs + 1.04 * raw + 2.26e-5 * g.d));
    if (route.tile == 0 || est < fused) {
      fused = est;
      route.tile = R;
    }
  }
  route.faster = route.tile != 0 && fused < 0.95 * layers;
  return route;
}

int64_t kouter_part_floats(const FlowGeom& g) {
  int64_t mn = 1;
  for (int l = 0; l < g.L; ++l)
    for (int i = 0; i <= g.nh; ++i) mn = std::max<int64_t>(mn, (int64_t)g.lin_out(l, i) * g.lin_in(l, i));
  int64_t s = (int64_t)(16 << 20) / mn;   // about 64 MB of partials at most
  if (s > kKouterMaxSlices) s = kKouterMaxSlices;
  if (s < 2) s = 2;
  return s * mn;
}

struct GradWs {
  int R, rb, ab, per_pair, slices;
  int64_t tiles, acts, gout, gaff, part, bpart, apart, total;
  WgradSlices z;
};

static GradWs grad_ws(const FlowGeom& g, int64_t n) {
  GradWs w{};
  const FlowShape s = flow_shape(g);
  w.R = flow_f32_grad_route(g, n).tile;
  w.tiles = (n + w.R - 1) / w.R;
  const int64_t rows = (n + 63) / 64 * 64;   // of the tiles, whatever their height
  auto al = [](int64_t v) { return (v + 63) / 64 * 64; };
  w.acts = al(s.act_base(g.L) * rows);
  w.gout = al(s.gcol(g.L, 0) * rows);
  w.gaff = al((int64_t)g.L * n * g.d);
  const int64_t pf = kouter_part_floats(g);
  int64_t most[2] = {0, 0};   // floats of a layer's partials, a bound that grows with n
  for (int l = 0; l < 2; ++l) {
    int64_t off = 0;
    for (int i = 0; i <= g.nh; ++i) {
      w.per_pair += wg_items(s, l, i);
      most[l] += kouter_most_slices(s.out(l, i), s.in(l, i), n, true, pf) * s.out(l, i) * s.in(l, i);
      w.z.count[l][i] = (int)kouter_slices(s.out(l, i), s.in(l, i), n, true, pf, &w.z.rows[l][i]);
      if (w.z.count[l][i] > w.slices) w.slices = w.z.count[l][i];
      w.z.part_off[l][i] = off;
      off += (int64_t)w.z.count[l][i] * s.out(l, i) * s.in(l, i);
    }
    w.z.part_layer[l] = off;
  }
  w.part = al((int64_t)(g.L / 2) * (most[0] + most[1]) + (g.L & 1) * most[0]);
  w.rb = colsum_blocks(n);
  w.bpart = al(s.gcol(g.L, 0) * w.rb);
  w.ab = affine_sum_blocks(n, g.d);
  w.apart = al((int64_t)g.L * w.ab * 2);
  w.total = w.acts + w.gout + w.gaff + w.part + w.bpart + w.apart;
  return w;
}

int64_t flow_f32_grad_floats(const FlowGeom& g, int64_t n) { return grad_ws(g, n).total; }

template <int K, int R>
static int launch_bwd(const FlowBwdArgs& a, size_t bytes, cudaStream_t st) {
  auto kern = k_flow_f32_bwd<K, R>;
  FMC_CUDA_TRY(allow_smem(kern, bytes));
  kern<<<(unsigned)a.tiles, FlowTile<R>::NT, bytes, st>>>(a);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}

template <int R>
static int launch_bwd_r(const FlowBwdArgs& a, size_t bytes, cudaStream_t st) {
#define CASE(k) \
  if (a.s.K == k) return launch_bwd<k, R>(a, bytes, st);
  CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(8) CASE(10) CASE(12) CASE(16)
#undef CASE
  set_error("n_bins=%d is not instantiated (2,3,4,5,6,8,10,12,16)", a.s.K);
  return FMC_ERR_UNSUPPORTED;
}

int flow_f32_grad(const FlowGeom& g, const float* theta, const float* aux, int64_t n, const float* save, float* ws,
                  float* grad, cudaStream_t st) {
  const GradWs w = grad_ws(g, n);
  FlowBwdArgs a{};
  const size_t bytes = bwd_smem(g, w.R, a);
  a.theta = theta;
  a.aux = aux;
  a.save = save;
  a.acts = ws;
  a.gout = ws + w.acts;
  a.gaff = a.gout + w.gout;
  float* part = a.gaff + w.gaff;
  float* bpart = part + w.part;
  float* apart = bpart + w.bpart;
  a.n = n;
  a.tiles = w.tiles;
  a.inv_n = 1.0f / (float)n;
  int rc = w.R == 64 ? launch_bwd_r<64>(a, bytes, st) : launch_bwd_r<16>(a, bytes, st);
  if (rc) return rc;
  WgradArgs b{};
  b.s = a.s;
  b.z = w.z;
  b.acts = a.acts;
  b.gout = a.gout;
  b.part = part;
  b.n = n;
  b.tiles = w.tiles;
  b.per_pair = w.per_pair;
  auto kw = w.R == 64 ? k_wgrad_f32<64> : k_wgrad_f32<16>;
  constexpr int wbytes = kWgStages * kWgStageFloats * 4;
  FMC_CUDA_TRY(cudaFuncSetAttribute(kw, cudaFuncAttributeMaxDynamicSharedMemorySize, wbytes));
  kw<<<dim3((unsigned)(w.per_pair * ((g.L + 1) / 2)), (unsigned)w.slices), kWgThreads, wbytes, st>>>(b);
  FMC_LAUNCH_CHECK();
  int64_t mx = 1;
  int mo = 1;
  for (int l = 0; l < 2; ++l)
    for (int i = 0; i <= g.nh; ++i) {
      mx = std::max<int64_t>(mx, (int64_t)a.s.out(l, i) * a.s.in(l, i));
      mo = std::max(mo, a.s.out(l, i));
    }
  const unsigned lin = (unsigned)(g.L * (g.nh + 1));
  k_sum_wgrad<<<dim3((unsigned)std::min<int64_t>((mx + 255) / 256, 64), lin), 256, 0, st>>>(a.s, w.z, part, grad);
  FMC_LAUNCH_CHECK();
  const dim3 bg((unsigned)((mo + 127) / 128), (unsigned)w.rb, lin);
  k_bias_partial<<<bg, 128, 0, st>>>(a.s, a.gout, n, w.tiles * w.R, (n + w.rb - 1) / w.rb, bpart);
  FMC_LAUNCH_CHECK();
  k_bias_final<<<dim3(bg.x, 1, lin), 128, 0, st>>>(a.s, bpart, w.rb, grad);
  FMC_LAUNCH_CHECK();
  k_affine_layers<<<dim3((unsigned)w.ab, (unsigned)g.L), 256, 0, st>>>(a.s, theta, save, a.gaff, n, apart);
  FMC_LAUNCH_CHECK();
  k_affine_final<<<(unsigned)g.L, 32, 0, st>>>(a.s, apart, w.ab, -a.inv_n * (float)g.d * (float)n, grad);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}

}  // namespace fmc
