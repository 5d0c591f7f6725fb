// targets.cuh -- registered target log-densities with hand-written adjoints.
//
// The reference takes an arbitrary JAX callable `logpdf(x, data)` and
// differentiates it with jax.value_and_grad (resource/kernel/MALA.py:59,
// resource/kernel/HMC.py:73-78). A fused device kernel cannot run Python, so
// the sampler is given a target descriptor (FmcTarget) and evaluates the
// value and its analytic gradient here.
//
// Work split: a chain is owned by a group of G lanes; lane `gl` holds the V
// consecutive coordinates j = gl*V + v (v < V) of the position. Coordinates
// j >= n_dim are padding: they hold 0, contribute 0 and get gradient 0.
// Reductions over coordinates are butterfly shuffles inside the group, so
// every lane of the group ends with the bitwise-same value.
#pragma once
#include "common.cuh"

namespace fmc {

constexpr int kMaxMixtureComponents = 16;

template <int V>
struct Vec { float v[V]; };

__device__ __forceinline__ float ldg_or(const float* p, int64_t i, float dflt) {
  return p ? __ldg(p + i) : dflt;
}

// Shared-memory copy of the diagonal-Gaussian / mixture tables: means [K][G V],
// inverse variances [K][G V] (missing tables get 0 and 1), log-weights [K].
// Rows are padded to the group's G * V coordinates with zeros (no contribution,
// zero gradient), so a lane reads its V entries without bounds or alignment
// checks.
__host__ __device__ inline int target_table_floats(int K, int w) { return 2 * K * w + K; }
template <int G, int V>
__device__ __forceinline__ void stage_target_table(const FmcTarget& t, float* tab) {
  constexpr int W = G * V;
  const int K = (t.kind == FMC_TARGET_GAUSS_MIXTURE) ? t.n_comp : 1;
  for (int i = threadIdx.x; i < K * W; i += blockDim.x) {
    const int k = i / W, j = i % W;
    const bool in = j < t.n_dim;
    tab[i] = (in && t.mean) ? __ldg(t.mean + k * t.n_dim + j) : 0.f;
    tab[K * W + i] = in ? (t.inv_var ? __ldg(t.inv_var + k * t.n_dim + j) : 1.f) : 0.f;
  }
  for (int k = threadIdx.x; k < K; k += blockDim.x) tab[2 * K * W + k] = t.log_w ? __ldg(t.log_w + k) : 0.f;
}

// this lane's V entries of one table row
template <int V>
__device__ __forceinline__ void tab_row(const float* row, int gl, float (&out)[V]) {
  if constexpr (V % 4 == 0) {
#pragma unroll
    for (int q = 0; q < V; q += 4) {
      const float4 t = *reinterpret_cast<const float4*>(row + gl * V + q);
      out[q] = t.x; out[q + 1] = t.y; out[q + 2] = t.z; out[q + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) out[v] = row[gl * V + v];
  }
}

// Quotient constants of a target, built once per kernel (the compiler does not
// move them out of the step loop by itself).
template <int TGT>
struct TargetConst {
  __device__ __forceinline__ explicit TargetConst(const FmcTarget&) {}
};
template <>
struct TargetConst<FMC_TARGET_DUAL_MOON> {
  ConstDiv by_s1, by_s3;
  bool fast;
  __device__ __forceinline__ explicit TargetConst(const FmcTarget& t)
      : by_s1(t.scalars[1]), by_s3(t.scalars[3]), fast(by_s1.in_range && by_s3.in_range) {}
};
template <>
struct TargetConst<FMC_TARGET_ROSENBROCK> {
  ConstDiv by_s0, by_half;
  int fast;   // 2: two-step quotients, 1: three corrections, 0: the division operator
  __device__ __forceinline__ explicit TargetConst(const FmcTarget& t)
      : by_s0(t.scalars[0]), by_half(0.5f * t.scalars[0]),
        fast(by_s0.in_range && by_half.in_range ? (by_s0.even ? 2 : 1) : 0) {}
};

// --------------------------------------------------------------- diag Gaussian
// tab: the shared-memory table (stage_target_table) or NULL for global loads
template <int G, int V, bool GRAD, bool VALUE>
__device__ __forceinline__ float tg_diag_gaussian(const FmcTarget& t, const float (&x)[V],
                                                  float (&g)[V], int gl, const float* tab) {
  const int d = t.n_dim;
  float s = 0.f;
  if (tab != nullptr) {
    float mu[V], iv[V];
    tab_row<V>(tab, gl, mu);
    tab_row<V>(tab + G * V, gl, iv);   // 0 on padding coordinates: no contribution
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const float dx = x[v] - mu[v];
      s += dx * dx * iv[v];
      if (GRAD) g[v] = -dx * iv[v];
    }
    return VALUE ? -0.5f * group_sum<G>(s) + t.scalars[0] : 0.f;
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int j = gl * V + v;
    if (j < d) {
      const float dx = x[v] - ldg_or(t.mean, j, 0.f);
      const float iv = ldg_or(t.inv_var, j, 1.f);
      s += dx * dx * iv;
      if (GRAD) g[v] = -dx * iv;
    } else if (GRAD) {
      g[v] = 0.f;
    }
  }
  return VALUE ? -0.5f * group_sum<G>(s) + t.scalars[0] : 0.f;
}

// --------------------------------------------------------------- dual moon
// log p = -0.5((|x| - s0)/s1)^2 + logsumexp(-0.5((x0 + s2)/s3)^2, -0.5((x0 - s2)/s3)^2)
template <int G, int V, bool GRAD, bool VALUE>
__device__ __forceinline__ float tg_dual_moon(const FmcTarget& t, const TargetConst<FMC_TARGET_DUAL_MOON>& tc,
                                              const float (&x)[V], float (&g)[V], int gl) {
  const int d = t.n_dim;
  const float s0 = t.scalars[0], s1 = t.scalars[1], s2 = t.scalars[2], s3 = t.scalars[3];
  float r2 = 0.f;
#pragma unroll
  for (int v = 0; v < V; ++v) r2 += x[v] * x[v];  // padding holds 0
  r2 = group_sum<G>(r2);
  const float r = sqrtf(r2);
  const float x0 = group_bcast<G>(x[0], 0);
  // quotients by s1 and s3: correctly rounded without a division each where
  // every numerator is in range, else the operator
  const ConstDiv &by_s1 = tc.by_s1, &by_s3 = tc.by_s3;
  const float na = x0 + s2, nb = x0 - s2, nr = r - s0;
  const bool fast = tc.fast && fminf(fminf(fabsf(na), fabsf(nb)), fabsf(nr)) >= 0x1p-25f &&
                    fmaxf(fmaxf(fabsf(na), fabsf(nb)), fabsf(nr)) <= 0x1p25f;
  float tt, za, zb, dtt = 0.f, dza = 0.f, dzb = 0.f;   // nr / s1, na / s3, nb / s3; -tt / s1, -za / s3, -zb / s3
  if (fast) {
    tt = by_s1(nr);
    za = by_s3(na);
    zb = by_s3(nb);
    if (GRAD) {
      dtt = -by_s1(tt);
      dza = by_s3(-za);
      dzb = by_s3(-zb);
    }
  } else {
    tt = nr / s1;
    za = na / s3;
    zb = nb / s3;
    if (GRAD) {
      dtt = -(tt / s1);
      dza = -za / s3;
      dzb = -zb / s3;
    }
  }
  const float a = -0.5f * za * za, b = -0.5f * zb * zb;
  const float m = fmaxf(a, b);
  const float lse = m + log1pf(expf(-fabsf(a - b)));
  if (GRAD) {
    const float cr = dtt / r;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int j = gl * V + v;
      g[v] = (j < d) ? cr * x[v] : 0.f;
    }
    if (gl == 0) {
      const float wa = expf(a - lse), wb = expf(b - lse);
      g[0] = __fadd_rn(g[0], __fmaf_rn(wb, dzb, __fmul_rn(wa, dza)));
    }
  }
  return -0.5f * tt * tt + lse;
}

// --------------------------------------------------------------- Gaussian mixture
// log p = logsumexp_k( log_w[k] - 0.5 sum_j (x_j - mean[k,j])^2 inv_var[k,j] )
// One pass over the components with an online log-sum-exp: running max m,
// running sum S = sum_k exp(e_k - m) and the running weighted gradient
// Gr = sum_k exp(e_k - m) * (-(x - mean_k) inv_var_k), rescaled whenever m
// grows; at the end lp = m + log S and grad = Gr / S. No per-component
// arrays, so the loop stays rolled and register use stays flat in K.
template <int G, int V, bool GRAD, bool VALUE>
__device__ __forceinline__ float tg_mixture(const FmcTarget& t, const float (&x)[V],
                                            float (&g)[V], int gl, const float* tab) {
  const int d = t.n_dim, K = t.n_comp;
  float m = -INFINITY, S = 0.f;
  float Gr[V];
#pragma unroll
  for (int v = 0; v < V; ++v) Gr[v] = 0.f;
  // one component's exponent and gradient into the running sums. e > m:
  // S = S w + 1, Gr = Gr w + gk and m = e; else S = S + w, Gr = Gr + w gk, with
  // w = e^-|e - m| (0 on the first component, m = -inf): operands picked
  // instead of a branch, because the chains of a warp disagree about it
  auto merge = [&](float e, const float (&gk)[V]) {
    const bool up = e > m;
    const float w = expf(-fabsf(e - m));
    S = fmaf(up ? S : 1.f, w, up ? 1.f : S);
    if (GRAD) {
#pragma unroll
      for (int v = 0; v < V; ++v) Gr[v] = fmaf(up ? Gr[v] : gk[v], w, up ? gk[v] : Gr[v]);
    }
    m = up ? e : m;
  };
  if (tab != nullptr) {
    // N components at a time: their sums over the coordinates are reduced
    // together (the shuffles of one hide the others' latency), then merged one
    // after the other
    constexpr int W = G * V;
    auto chunk = [&](auto n_comps, int k0) {
      constexpr int N = decltype(n_comps)::value;
      float q[N], gk[N][V];
#pragma unroll
      for (int n = 0; n < N; ++n) {
        float mu[V], iv[V];
        tab_row<V>(tab + (k0 + n) * W, gl, mu);
        tab_row<V>(tab + (K + k0 + n) * W, gl, iv);   // 0 on padding coordinates
        q[n] = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const float dx = x[v] - mu[v];
          q[n] += dx * dx * iv[v];
          gk[n][v] = -dx * iv[v];
        }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        float w[N];
#pragma unroll
        for (int n = 0; n < N; ++n) w[n] = __shfl_xor_sync(0xffffffffu, q[n], o, G);
#pragma unroll
        for (int n = 0; n < N; ++n) q[n] += w[n];
      }
#pragma unroll
      for (int n = 0; n < N; ++n) merge(tab[2 * K * W + k0 + n] - 0.5f * q[n], gk[n]);
    };
    constexpr int NC = V <= 4 ? 4 : 2;
    int k = 0;
#pragma unroll 1
    for (; k + NC <= K; k += NC) chunk(IntC<NC>{}, k);
#pragma unroll 1
    for (; k < K; ++k) chunk(IntC<1>{}, k);
  } else {
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
      float q = 0.f, gk[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int j = gl * V + v;
        gk[v] = 0.f;
        if (j < d) {
          const float dx = x[v] - ldg_or(t.mean, (int64_t)k * d + j, 0.f);
          const float iv = ldg_or(t.inv_var, (int64_t)k * d + j, 1.f);
          q += dx * dx * iv;
          gk[v] = -dx * iv;
        }
      }
      merge(ldg_or(t.log_w, k, 0.f) - 0.5f * group_sum<G>(q), gk);
    }
  }
  if (GRAD) {
    const float inv = 1.f / S;
#pragma unroll
    for (int v = 0; v < V; ++v) g[v] = Gr[v] * inv;
  }
  return VALUE ? m + logf(S) : 0.f;
}

// --------------------------------------------------------------- Rosenbrock chain
// log p = -sum_{i=0}^{d-2} [ (s1 - x_i)^2 / s0 + s2 (x_{i+1} - x_i^2)^2 ]
template <int G, int V, bool GRAD, bool VALUE>
__device__ __forceinline__ float tg_rosenbrock(const FmcTarget& t, const TargetConst<FMC_TARGET_ROSENBROCK>& tc,
                                               const float (&x)[V], float (&g)[V], int gl) {
  const int d = t.n_dim;
  const float s0 = t.scalars[0], s1 = t.scalars[1], s2 = t.scalars[2];
  // neighbours across the lane boundary
  const float next_first = __shfl_down_sync(0xffffffffu, x[0], 1, G);   // x_{gl*V+V}
  const float prev_last = __shfl_up_sync(0xffffffffu, x[V - 1], 1, G);  // x_{gl*V-1}
  float a[V], lo, hi;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    a[v] = s1 - x[v];
    const float m = fabsf(a[v]);
    lo = v ? fminf(lo, m) : m;
    hi = v ? fmaxf(hi, m) : m;
  }
  // quotients by s0: 2 a / s0 (as a / (s0 / 2)) for the gradient, a^2 / s0 for
  // the value; correctly rounded on every path
  const ConstDiv &by_s0 = tc.by_s0, &by_half = tc.by_half;
  const bool fast = lo >= 0x1p-29f && hi <= 0x1p29f;
  float q1[V], q2[V];
  if (fast && tc.fast == 2) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (GRAD) q1[v] = by_half.two(a[v]);
      if (VALUE) q2[v] = by_s0.two(a[v] * a[v]);
    }
  } else if (fast && tc.fast == 1) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (GRAD) q1[v] = by_half(a[v]);
      if (VALUE) q2[v] = by_s0(a[v] * a[v]);
    }
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (GRAD) q1[v] = 2.f * a[v] / s0;
      if (VALUE) q2[v] = a[v] * a[v] / s0;
    }
  }
  // coordinate j has a successor term (j + 1 < d) and a predecessor term
  // (1 <= j < d). Where d is a multiple of V a lane is wholly inside or wholly
  // padding and only its first and last coordinate differ from the others.
  const bool whole = d % V == 0;
  const bool in = gl * V < d, last_next = (gl + 1) * V < d, first_prev = in && gl > 0;
  float s = 0.f;
  auto combine = [&](auto by_lane) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int j = gl * V + v;
      const float xn = (v + 1 < V) ? x[v + 1] : next_first;
      const float xp = (v > 0) ? x[v - 1] : prev_last;
      const bool has_next = decltype(by_lane)::value ? (v + 1 < V ? in : last_next) : j + 1 < d;
      const bool has_prev = decltype(by_lane)::value ? (v > 0 ? in : first_prev) : j >= 1 && j < d;
      const float b = xn - x[v] * x[v];
      if (VALUE && has_next) s += q2[v] + s2 * b * b;
      if (GRAD) {
        float gv = has_next ? q1[v] + 4.f * s2 * x[v] * b : 0.f;
        if (has_prev) gv -= 2.f * s2 * (x[v] - xp * xp);
        g[v] = gv;
      }
    }
  };
  if (whole) combine(IntC<1>{});
  else combine(IntC<0>{});
  return VALUE ? -group_sum<G>(s) : 0.f;
}

// --------------------------------------------------------------- dense Gaussian
// log p = -0.5 (x-m)^T P (x-m) + scalars[0], P symmetric (the host symmetrises).
// The group stages dx in shared memory (`stage`, n_dim floats per group).
template <int G, int V, bool GRAD, bool VALUE>
__device__ __forceinline__ float tg_dense_gaussian(const FmcTarget& t, const float (&x)[V],
                                                   float (&g)[V], int gl, float* stage) {
  const int d = t.n_dim;
  float dx[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int j = gl * V + v;
    dx[v] = (j < d) ? x[v] - ldg_or(t.mean, j, 0.f) : 0.f;
    if (j < d) stage[j] = dx[v];
  }
  __syncwarp();
  float acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.f;
  for (int k = 0; k < d; ++k) {
    const float dk = stage[k];
    const float* row = t.precision + (int64_t)k * d;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int j = gl * V + v;
      if (j < d) acc[v] += __ldg(row + j) * dk;  // P[k, j] = P[j, k]
    }
  }
  __syncwarp();
  float s = 0.f;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    s += dx[v] * acc[v];
    if (GRAD) g[v] = -acc[v];
  }
  return VALUE ? -0.5f * group_sum<G>(s) + t.scalars[0] : 0.f;
}

// stage: the dense Gaussian's per-group scratch (n_dim floats), or for the
// diagonal Gaussian and the mixture the block's shared-memory table copy
// (stage_target_table; NULL = read the tables from global memory).
// VALUE = false: only the gradient is wanted and 0 is returned (the compiler
// keeps the shuffles of an unused reduction: 128-D Rosenbrock HMC, 16 of 17
// evaluations, 2.17 -> 1.52 ms)
template <int TGT, int G, int V, bool GRAD, bool VALUE = true>
__device__ __forceinline__ float target_eval(const FmcTarget& t, const TargetConst<TGT>& tc, const float (&x)[V],
                                             float (&g)[V], int gl, float* stage) {
  if constexpr (TGT == FMC_TARGET_DIAG_GAUSSIAN) return tg_diag_gaussian<G, V, GRAD, VALUE>(t, x, g, gl, stage);
  else if constexpr (TGT == FMC_TARGET_DUAL_MOON) return tg_dual_moon<G, V, GRAD, VALUE>(t, tc, x, g, gl);
  else if constexpr (TGT == FMC_TARGET_GAUSS_MIXTURE) return tg_mixture<G, V, GRAD, VALUE>(t, x, g, gl, stage);
  else if constexpr (TGT == FMC_TARGET_ROSENBROCK) return tg_rosenbrock<G, V, GRAD, VALUE>(t, tc, x, g, gl);
  else return tg_dense_gaussian<G, V, GRAD, VALUE>(t, x, g, gl, stage);
}

}  // namespace fmc
