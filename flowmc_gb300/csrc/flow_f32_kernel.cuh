// flow_f32_kernel.cuh -- MaskedCouplingRQSpline passes in FP32 as one launch: every
// layer's ScalarAffine, conditioner MLP and spline for a tile of rows
// (rqSpline.py:450-504, common.py:127-168, 211-240).
//
// Before, a pass was five launches per layer (affine, three 64 x 64-tile SIMT
// GEMMs, spline) with the [rows, n_t (3K + 1)] conditioner outputs written to
// HBM and read back by a spline kernel whose lanes strode 3K + 1 floats. Here
// activations and outputs stay in shared memory and a row's log-determinant is
// summed in the order the launches had. Same bits, apart from the last place of
// some log-determinants. Bound by FMA issue (packed FMAs with one operand in both
// halves run at about 62 of the 80 TFLOP/s FP32 peak here) and, beside it, the
// latency of the spline and tanh phases with eight warps per SM. Measured on
// GB300: log_prob of 100,003 rows, 32-D, 8 x [128, 128] x 10 bins, 6.00 -> 3.64 ms
// (37 TFLOP/s); the two passes of a 20-chain x 30-step global step of the 5-D 4 x
// [32, 32] flow, 45 launches -> 2, 274 -> 89 us for the whole step.
#pragma once
#include "flow_f32.cuh"
#include "flow_f32.h"

namespace fmc {

struct FlowF32Args {
  FlowShape s;
  const float* theta;
  const float* aux;
  const float* x;      // [n, d] input rows (unused with in_mode FLOW_IN_BASE)
  const float* z;      // FLOW_IN_BASE: explicit base normals [n, d] or NULL
  Rng rng;             // FLOW_IN_BASE: Philox stream
  int64_t n;
  int in_mode, out_mode;
  float* y;            // [n, d] (FLOW_OUT_ROWS, FLOW_OUT_DATA)
  float* ld;           // [n] or NULL (FLOW_OUT_ROWS, FLOW_OUT_LOGP)
  float* logp;         // [n] (FLOW_OUT_LOGP)
  // SAVE (training): [L + 1, n, d], every layer's input and the output
  float* save;
  float* acts;         // and every layer's activations in tiles of R rows: [layer][array][tile][column][R]
  int64_t tiles;
  int ldx, cond_floats, act_floats;   // pitch of the row tile; sizes of the conditioning block and an activation buffer
};

// shared memory (floats): xs [R][ldx]; cond [nc][R + 4], whose place the splines'
// log-dets [32][R] take afterwards; two activation buffers [H][R + 4], of
// which the one the last Linear does not read holds its output tile; weight
// stages; per-thread log-det partials [256]
template <int K, int R, bool INV, bool SAVE>
__global__ void __launch_bounds__(FlowTile<R>::NT, 2) k_flow_f32(const __grid_constant__ FlowF32Args a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int P = 3 * K + 1;
  using T = FlowTile<R>;
  constexpr int NT = T::NT, NW = NT / 32;
  const FlowShape& s = a.s;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int d = s.d;
  float* xs = sm;
  float* cond = xs + R * a.ldx;
  float* act0 = cond + a.cond_floats;
  float* act1 = act0 + a.act_floats;
  float* ring = act1 + a.act_floats;
  float* part = ring + T::ST * kFlowStageFloats;
  const int r0 = (wid / T::WC) * 32 + flow_lane_row();
  const int c0 = (wid % T::WC) * (8 * T::TN) + flow_lane_col();
  const int64_t row_base = (int64_t)blockIdx.x * R;
  const int rows = (int)(a.n - row_base < R ? a.n - row_base : R);

  WStream<T::NT, T::ST> w;
  w.begin(&s, a.theta, ring, INV);
  int slot = 0;

  // ---- input rows (zeros past n)
  const Rng rng = a.rng.at_epoch();
  for (int r = wid; r < R; r += NW) {
    const int64_t gr = row_base + r;
    for (int j = lane; j < d; j += 32) {
      float v = 0.f;
      if (r < rows) {
        if (a.in_mode == FLOW_IN_BASE) {
          // jax.random.multivariate_normal(0, c I): sqrt(c) z
          if (a.z) {
            v = a.z[gr * d + j];
          } else {
            const u32x4 b = rng.draw((uint64_t)gr, 0, (uint32_t)(j >> 1), RNG_TAG_NF_NORMAL);
            float z0, z1;
            box_muller(b.x, b.y, z0, z1);
            v = (j & 1) ? z1 : z0;
          }
          v = v * sqrtf(a.aux[2 * d]);
        } else {
          v = a.x[gr * d + j];
          if (a.in_mode == FLOW_IN_DATA) v = (v - a.aux[j]) / sqrtf(a.aux[d + j]);
        }
      }
      xs[r * a.ldx + j] = v;
    }
  }
  float ld = 0.f;   // of row tid (tid < R)

  for (int u = 0; u < s.L; ++u) {
    const int l = INV ? s.L - 1 - u : u;
    const float* th = a.theta + s.layer_off(l);
    const int nc = s.nc(l), nt = s.nt(l), cpar = s.cpar(l), tpar = s.tpar(l);
    __syncthreads();   // xs and the log-det partials are complete
    // ---- ScalarAffine; the conditioning coordinates, zero padded, into cond
    {
      const float sc = __ldg(th), sh = __ldg(th + 1);
      const float es = expf(INV ? -sc : sc);
      const int kp = (nc + 15) & ~15;
      for (int r = wid; r < R; r += NW) {
        float* xr = xs + r * a.ldx;
        for (int j = lane; j < d; j += 32) {
          const float v0 = xr[j];
          if (SAVE && r < rows) a.save[((int64_t)u * a.n + row_base + r) * d + j] = v0;
          const float v = scalar_affine(v0, es, sh, INV ? 1 : 0);
          xr[j] = v;
          if ((j & 1) == cpar) cond[(j >> 1) * T::LD + r] = v;
        }
        for (int k = nc + lane; k < kp; k += 32) cond[k * T::LD + r] = 0.f;
      }
      if (tid < R) {
        const float al = scalar_affine_logdet(sc, d, INV ? 1 : 0);
        ld = u == 0 ? al : __fadd_rn(ld, al);
      }
    }
    // SAVE: a tile of the layer's array i to the saved activations
    auto keep = [&](const float* tile, int i, int first, int cols, int of) {
      fence_async();
      __syncthreads();
      tile_store<R>(tile, a.acts + ((s.act_base(l) + s.act_col(l, i)) * a.tiles + (int64_t)blockIdx.x * of + first) * R,
                    cols);
    };
    if (SAVE) {
      bulk_store_wait<0>();   // the previous layer's last tile
      keep(cond, 0, 0, nc, nc);
    }
    // ---- hidden Linears
    const float* A = cond;
    float* cur = act0;
    float* other = act1;
    for (int i = 0; i < s.nh; ++i) {
      const int in = s.in(l, i), out = s.out(l, i);
      const float* bias = th + s.w_off(l, i) + (int64_t)out * in;
      const int op = (out + 15) & ~15;
      for (int n0 = 0; n0 < out; n0 += kFlowCols) {
        const int N = min(kFlowCols, out - n0);
        float4 v[T::TQ][T::TN];
        // every tile but the newest kept one has been read; the product's
        // barriers order that before the writes below
        if (SAVE) bulk_store_wait<1>();
        flow_product<R>(w, ring, slot, A, N, in, r0, c0, v);
        // biased sums to shared memory, then tanh on the thread's own values in a
        // rolled loop (64 inlined tanh would be most of the kernel's code)
#pragma unroll
        for (int j = 0; j < T::TN; ++j) {
          const int c = n0 + c0 + 8 * j;
          if (c < op) {
            const float b = c < out ? __ldg(bias + c) : 0.f;
#pragma unroll
            for (int q = 0; q < T::TQ; ++q) {
              const float4 t = v[q][j];
              *reinterpret_cast<float4*>(cur + c * T::LD + r0 + 16 * q) =
                  make_float4(t.x + b, t.y + b, t.z + b, t.w + b);
            }
          }
        }
#pragma unroll 1
        for (int j = 0; j < T::TN; ++j) {
          const int c = n0 + c0 + 8 * j;
          if (c >= op) break;
          const bool on = c < out;
#pragma unroll
          for (int q = 0; q < T::TQ; ++q) {
            float4* p = reinterpret_cast<float4*>(cur + c * T::LD + r0 + 16 * q);
            const float4 t = *p;
            const float4 h = on ? make_float4(tanhf(t.x), tanhf(t.y), tanhf(t.z), tanhf(t.w))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
            *p = h;
          }
        }
      }
      if (SAVE) keep(cur, i + 1, 0, out, out);
      A = cur;
      float* t = cur;
      cur = other;
      other = t;
    }
    // ---- last Linear, a group of coordinates at a time, and their splines
    const int row = tid % R;
    const int in = s.in(l, s.nh), out = nt * P, tc = s.dg * P;
    const float* bias = th + s.w_off(l, s.nh) + (int64_t)out * in;
    float* raw = cur;
    float* lb = cond;   // [32][R]: log-dets of coordinates t = k mod 32, summed in t order
    for (int n0 = 0, t0 = 0; n0 < out; n0 += tc, t0 += s.dg) {
      const int N = min(tc, out - n0);
      {
        float4 v[T::TQ][T::TN];
        if (SAVE) {
          if (t0 == 0) bulk_store_wait<1>();
          else bulk_store_wait<0>();   // the previous group's tile
        }
        flow_product<R>(w, ring, slot, A, N, in, r0, c0, v);
#pragma unroll
        for (int j = 0; j < T::TN; ++j) {
          const int c = c0 + 8 * j;
          if (c < N) {
            const float b = __ldg(bias + n0 + c);
#pragma unroll
            for (int q = 0; q < T::TQ; ++q) {
              const float4 t = v[q][j];
              const float4 o = make_float4(t.x + b, t.y + b, t.z + b, t.w + b);
              *reinterpret_cast<float4*>(raw + c * T::LD + r0 + 16 * q) = o;
            }
          }
        }
      }
      if (t0 == 0)
        for (int e = tid; e < 32 * R; e += NT) lb[e] = 0.f;
      if (SAVE) keep(raw, s.nh + 1, n0, N, out);
      else __syncthreads();
      const int items = (N / P) * R;
      for (int e = tid; e < items; e += NT) {
        const int t = e / R;
        float prm[P];
#pragma unroll
        for (int p = 0; p < P; ++p) prm[p] = raw[(t * P + p) * T::LD + row];
        float* xp = xs + row * a.ldx + 2 * (t0 + t) + tpar;
        float o, lv;
        rqs_apply<K, INV>(prm, *xp, s.cfg, o, lv);
        *xp = o;
        lb[((t0 + t) & 31) * R + row] += lv;
      }
    }
    // the row's log-det: the 32 sums as one balanced tree (the order of a warp
    // butterfly over the coordinates), NQ threads per row
    __syncthreads();
    {
      constexpr int NQ = NT / R, M = 32 / NQ;
      const int q = tid / R;
      float v[M];
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] = lb[(q + NQ * m) * R + row];
#pragma unroll
      for (int h = M / 2; h > 0; h >>= 1)
#pragma unroll
        for (int m = 0; m < h; ++m) v[m] += v[m + h];
      part[tid] = v[0];
      __syncthreads();
      if (tid < R) {
        float p[NQ];
#pragma unroll
        for (int m = 0; m < NQ; ++m) p[m] = part[m * R + tid];
#pragma unroll
        for (int h = NQ / 2; h > 0; h >>= 1)
#pragma unroll
          for (int m = 0; m < h; ++m) p[m] += p[m + h];
        ld = __fadd_rn(ld, p[0]);
      }
    }
  }
  if (SAVE) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // shared memory outlives the copies
  // ---- results
  if (a.out_mode == FLOW_OUT_LOGP) {
    __syncthreads();   // the sums above have read part
    if (tid < R) part[tid] = ld;
    __syncthreads();
    const float c = a.aux[2 * d];
    for (int r = wid; r < rows; r += NW) {
      const int64_t gr = row_base + r;
      float q = 0.f;
      for (int j = lane; j < d; j += 32) {
        const float v = xs[r * a.ldx + j];
        if (SAVE) a.save[((int64_t)s.L * a.n + gr) * d + j] = v;
        q += v * v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      // multivariate_normal.logpdf(y, 0, c I) (common.py:285-286)
      if (lane == 0) a.logp[gr] = part[r] + (-0.5f * q / c - 0.5f * (float)d * logf(6.283185307179586f * c));
    }
  } else {
    for (int r = wid; r < rows; r += NW) {
      const int64_t gr = row_base + r;
      for (int j = lane; j < d; j += 32) {
        float v = xs[r * a.ldx + j];
        if (a.out_mode == FLOW_OUT_DATA) v = v * sqrtf(a.aux[d + j]) + a.aux[j];
        a.y[gr * d + j] = v;
      }
    }
    if (a.ld != nullptr && tid < rows) a.ld[row_base + tid] = ld;
  }
}

template <int K, int R, bool INV, bool SAVE>
static int launch_k(const FlowF32Args& a, size_t bytes, cudaStream_t st) {
  auto kern = k_flow_f32<K, R, INV, SAVE>;
  FMC_CUDA_TRY(allow_smem(kern, bytes));
  kern<<<(unsigned)((a.n + R - 1) / R), FlowTile<R>::NT, bytes, st>>>(a);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}

// one direction and tile height, for the instantiated bin counts
template <int R, bool INV, bool SAVE>
static int launch_r(const FlowF32Args& a, size_t bytes, cudaStream_t st) {
#define CASE(k) \
  if (a.s.K == k) return launch_k<k, R, INV, SAVE>(a, bytes, st);
  CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(8) CASE(10) CASE(12) CASE(16)
#undef CASE
  set_error("n_bins=%d is not instantiated (2,3,4,5,6,8,10,12,16)", a.s.K);
  return FMC_ERR_UNSUPPORTED;
}

// compiled apart (flow_f32_fwd.cu, flow_f32_inv.cu, flow_f32_save.cu)
int launch_flow_f32_fwd(const FlowF32Args& a, int R, size_t bytes, cudaStream_t st);
int launch_flow_f32_inv(const FlowF32Args& a, int R, size_t bytes, cudaStream_t st);
int launch_flow_f32_save(const FlowF32Args& a, int R, size_t bytes, cudaStream_t st);

}  // namespace fmc
