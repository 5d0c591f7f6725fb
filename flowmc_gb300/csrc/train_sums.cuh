// train_sums.cuh -- fixed-order sums over the batch shared by the flow training
// paths (flow_train.cu, flow_f32_bwd.cu), so that both add in the same order.
#pragma once
#include "common.cuh"

namespace fmc {

// row blocks of a column sum over n rows
inline int colsum_blocks(int64_t n) {
  int64_t rb = (n + 511) / 512;
  if (rb > 128) rb = 128;
  return (int)(rb < 1 ? 1 : rb);
}

// blocks of the ScalarAffine adjoint over n rows of d coordinates
inline int affine_sum_blocks(int64_t n, int d) {
  int64_t b = (n * d + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 8;
  if (b > cap) b = cap;
  if (b > 1024) b = 1024;
  return (int)(b < 1 ? 1 : b);
}

template <int NT>
__device__ __forceinline__ float block_sum(float v, float* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  float r = 0.f;
  if (threadIdx.x < 32) {
    r = (lane < NT / 32) ? sh[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  }
  return r;  // valid in thread 0
}

// Per-block sums (256 threads) of gv = g * es and g * x over all rows: one warp
// per row, rows strided over the grid. get(r, j, g, x, gv) gives the values (gv
// rounded, __fmul_rn: the compiler would fold the product into the sum where it
// is not stored, and the two paths would differ in the last place).
template <typename F>
__device__ __forceinline__ void affine_sums(int64_t n, int d, float* part, F get) {
  __shared__ float sh[32];
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  float st = 0.f, ss = 0.f;
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps)
    for (int j = lane; j < d; j += 32) {
      float g, x, gv;
      get(r, j, g, x, gv);
      st += gv;
      ss = __fmaf_rn(g, x, ss);
    }
  st = block_sum<256>(st, sh);
  ss = block_sum<256>(ss, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = st;
    part[2 * blockIdx.x + 1] = ss;
  }
}

// affine_sums with the loads of a row's four coordinates per lane issued
// ahead of their use: load(r, j, g, x), then gv = use(r, j, g), in the same order
template <typename L, typename U>
__device__ __forceinline__ void affine_sums_ahead(int64_t n, int d, float* part, L load, U use) {
  __shared__ float sh[32];
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  float st = 0.f, ss = 0.f;
  auto add = [&](int64_t r, int j, float g, float x) {
    st += use(r, j, g);
    ss = __fmaf_rn(g, x, ss);
  };
  int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (; r < n; r += warps)
    for (int j0 = lane; j0 < d; j0 += 128) {
      float g[4], x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j0 + 32 * k < d) load(r, j0 + 32 * k, g[k], x[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j0 + 32 * k < d) add(r, j0 + 32 * k, g[k], x[k]);
    }
  st = block_sum<256>(st, sh);
  ss = block_sum<256>(ss, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = st;
    part[2 * blockIdx.x + 1] = ss;
  }
}

// the ScalarAffine's two gradients from the nb block partials: one warp,
// lane i summing partials i, i + 32, ..., then a fixed-order butterfly
__device__ __forceinline__ void affine_param_grad(const float* __restrict__ part, int nb, float ld_term,
                                                  float* __restrict__ g_layer) {
  const int lane = threadIdx.x & 31;
  float st = 0.f, ss = 0.f;
  for (int b = lane; b < nb; b += 32) {
    st += part[2 * b];
    ss += part[2 * b + 1];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    st += __shfl_xor_sync(0xffffffffu, st, o);
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
  }
  if (lane == 0) {
    g_layer[0] = ss + ld_term;  // d/d scale
    g_layer[1] = st;            // d/d shift
  }
}

}  // namespace fmc
