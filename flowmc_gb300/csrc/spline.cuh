// spline.cuh -- rational-quadratic spline (forward, inverse, adjoint) for one
// coordinate, templated on the bin count K.
//
// Follows flowMC's rqSpline.py:
//   knots     _normalize_bin_sizes / _normalize_knot_slopes / get_params  (:20-39, :310-338)
//   forward   _rational_quadratic_spline_fwd (:42-128)
//   inverse   _safe_quadratic_root + _rational_quadratic_spline_inv (:131-239)
// The bin is picked while the knots run by with compile-time indices, so every
// array stays in registers. The adjoint is written out by hand: through the
// spline formula, the selected bin's knots, the cumulative sums, the two
// softmaxes and the softplus slopes.
#pragma once
#include <cuda_bf16.h>
#include "common.cuh"

namespace fmc {

struct SplineCfg {
  float rmin, rmax, min_bin, min_slope, slope_offset;
};

__device__ __forceinline__ float softplus_f(float a) {
  // jax.nn.softplus = logaddexp(a, 0)
  return fmaxf(a, 0.f) + log1pf(expf(-fabsf(a)));
}

// softmax numerators e^(r - max) and their sum
template <int K>
__device__ __forceinline__ float softmax_num(const float* r, float (&p)[K]) {
  float m = r[0];
#pragma unroll
  for (int k = 1; k < K; ++k) m = fmaxf(m, r[k]);
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    p[k] = expf(r[k] - m);
    s += p[k];
  }
  return s;
}

// p[k] / s for every k, correctly rounded: one reciprocal and five FMA-pipe
// steps each where the smallest numerator allows (s is 1 .. K), else the
// division operator
template <int K>
__device__ __forceinline__ void softmax_div(float (&p)[K], float s) {
  float lo = p[0];
#pragma unroll
  for (int k = 1; k < K; ++k) lo = fminf(lo, p[k]);
  if (lo >= 0x1p-60f) {
    const MarkDiv by(s);
#pragma unroll
    for (int k = 0; k < K; ++k) p[k] = by(p[k]);
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k) p[k] = p[k] / s;
  }
}

// The spline (or its inverse) at v and the log-determinant. raw: the 3K+1
// conditioner outputs of one coordinate. The knots run on while the bin that
// holds v is carried along, and only the bin's two slopes (in the tails the end
// slope) go through the softplus.
template <int K, bool INV>
__device__ __forceinline__ void rqs_apply(const float (&raw)[3 * K + 1], float v, const SplineCfg& c, float& out,
                                          float& ld) {
  const float scale = (c.rmax - c.rmin) - (float)K * c.min_bin;
  float pw[K], ph[K];
  softmax_div<K>(pw, softmax_num<K>(raw, pw));
  softmax_div<K>(ph, softmax_num<K>(raw + K, ph));
  const bool below = v <= c.rmin, above = v >= c.rmax;
  // bin 0 also covers "no bin" (rqSpline.py:70-72)
  float cw = 0.f, ch = 0.f, xk = c.rmin, yk = c.rmin;   // running left knot
  float x0 = c.rmin, y0 = c.rmin, x1 = c.rmax, y1 = c.rmax, r0 = raw[2 * K], r1 = raw[2 * K + 1];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float xn = c.rmax, yn = c.rmax;   // right knot of bin k
    if (k < K - 1) {
      cw += pw[k] * scale + c.min_bin;
      ch += ph[k] * scale + c.min_bin;
      xn = c.rmin + cw;
      yn = c.rmin + ch;
    }
    const bool in = k == 0 || (INV ? v >= yk && v < yn : v >= xk && v < xn);
    if (in) {
      x0 = xk; x1 = xn; y0 = yk; y1 = yn;
      r0 = raw[2 * K + k];
      r1 = raw[2 * K + k + 1];
    }
    xk = xn;
    yk = yn;
  }
  if (above) r1 = raw[3 * K];
  const float d0 = softplus_f(r0 + c.slope_offset) + c.min_slope;
  const float d1 = softplus_f(r1 + c.slope_offset) + c.min_slope;
  const float w = x1 - x0, h = y1 - y0;
  const float s = h / w;
  const float st = d1 + d0 - 2.f * s;
  float z;
  if (!INV) {
    z = fminf(fmaxf((v - x0) / w, 0.f), 1.f);
  } else {
    const float ww = fminf(fmaxf((v - y0) / h, 0.f), 1.f);
    const float cq = -s * ww;
    const float bq = d0 - st * ww;
    const float aq = s - bq;
    // _safe_quadratic_root (rqSpline.py:131-155)
    const float disc = bq * bq - 4.f * aq * cq;
    float sqd = sqrtf(fmaxf(disc, 1.17549435e-38f));
    if (!(disc > 0.f)) sqd = 0.f;
    const float num = (bq >= 0.f) ? 2.f * cq : -bq + sqd;
    const float dnm = (bq >= 0.f) ? -bq - sqd : 2.f * aq;
    z = fminf(fmaxf(num / dnm, 0.f), 1.f);
  }
  const float sq = z * z, q = z - sq, om = 1.f - z, sq1 = om * om;
  const float den = s + st * q;
  const float A = fmaf(d0, sq1, fmaf(d1, sq, __fmul_rn(2.f * s, q)));
  if (!INV) {
    const float num = h * (s * sq + d0 * q);
    out = y0 + num / den;
    ld = 2.f * logf(s) + logf(A) - 2.f * logf(den);
    if (below) { out = (v - c.rmin) * d0 + c.rmin; ld = logf(d0); }
    if (above) { out = (v - c.rmax) * d1 + c.rmax; ld = logf(d1); }
  } else {
    out = w * z + x0;
    ld = -2.f * logf(s) - logf(A) + 2.f * logf(den);
    if (below) { out = (v - c.rmin) / d0 + c.rmin; ld = -logf(d0); }
    if (above) { out = (v - c.rmax) / d1 + c.rmax; ld = -logf(d1); }
  }
}

// Adjoint of (y, ld) = rqs_apply<K, false>(x; raw): given gy = dL/dy and gl =
// dL/dld, returns dL/dx, and put(p, v) receives dL/draw[p]. Organised around the
// bin that holds x: only its two knots carry gradient into the cumulative widths
// and heights, and only its two slopes (in a tail the end slope) through the
// softplus.
template <int K, typename F>
__device__ __forceinline__ float rqs_adjoint(const float (&raw)[3 * K + 1], float x, const SplineCfg& c, float gy,
                                             float gl, F put) {
  const float scale = (c.rmax - c.rmin) - (float)K * c.min_bin;
  float pw[K], ph[K];
  softmax_div<K>(pw, softmax_num<K>(raw, pw));
  softmax_div<K>(ph, softmax_num<K>(raw + K, ph));
  const bool below = x <= c.rmin, above = x >= c.rmax;
  float cw = 0.f, ch = 0.f, xk = c.rmin, yk = c.rmin;
  float x0 = c.rmin, y0 = c.rmin, x1 = c.rmax, y1 = c.rmax, r0 = raw[2 * K], r1 = raw[2 * K + 1];
  int kb = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float xn = c.rmax, yn = c.rmax;
    if (k < K - 1) {
      cw += pw[k] * scale + c.min_bin;
      ch += ph[k] * scale + c.min_bin;
      xn = c.rmin + cw;
      yn = c.rmin + ch;
    }
    if (k == 0 || (x >= xk && x < xn)) {
      x0 = xk; x1 = xn; y0 = yk; y1 = yn;
      r0 = raw[2 * K + k];
      r1 = raw[2 * K + k + 1];
      kb = k;
    }
    xk = xn;
    yk = yn;
  }
  int k0 = kb, k1 = kb + 1;   // the slopes with gradients g_d0, g_d1
  if (above) {
    r1 = raw[3 * K];
    k1 = K;
  }
  const float d0 = softplus_f(r0 + c.slope_offset) + c.min_slope;
  const float d1 = softplus_f(r1 + c.slope_offset) + c.min_slope;
  float gx, g_x0 = 0.f, g_x1 = 0.f, g_y0 = 0.f, g_y1 = 0.f, g_d0 = 0.f, g_d1 = 0.f;
  if (below) {
    gx = gy * d0;
    g_d0 = gy * (x - c.rmin) + gl / d0;
    k1 = -1;
  } else if (above) {
    gx = gy * d1;
    g_d1 = gy * (x - c.rmax) + gl / d1;
    k0 = -1;
  } else {
    const float w = x1 - x0, h = y1 - y0;
    const float s = h / w;
    const float zr = (x - x0) / w;
    const float z = fminf(fmaxf(zr, 0.f), 1.f);
    const float sq = z * z, q = z - sq, om = 1.f - z, sq1 = om * om;
    const float st = d1 + d0 - 2.f * s;
    const float num = h * (s * sq + d0 * q);
    const float den = s + st * q;
    const float A = fmaf(d0, sq1, fmaf(d1, sq, __fmul_rn(2.f * s, q)));
    // y = y0 + num/den ; ld = 2 log s + log A - 2 log den
    const float g_num = gy / den;
    const float g_den = -gy * num / (den * den) - 2.f * gl / den;
    const float g_A = gl / A;
    float g_s = 2.f * gl / s;
    float g_h = g_num * (s * sq + d0 * q);
    g_s += g_num * h * sq;
    g_s += g_den * (1.f - 2.f * q);
    g_s += g_A * 2.f * q;
    // sums of products with the rounding of each spelled out
    const float nh = __fmul_rn(g_num, h);
    g_d0 = fmaf(g_A, sq1, fmaf(nh, q, __fmul_rn(g_den, q)));
    g_d1 = fmaf(g_A, sq, __fmul_rn(g_den, q));
    const float g_q = fmaf(g_A * 2.f, s, fmaf(nh, d0, __fmul_rn(g_den, st)));
    const float g_sq = fmaf(nh, s, __fmul_rn(g_A, d1));
    const float g_z =
        fmaf(__fmul_rn(-g_A, d0) * 2.f, om, fmaf(g_sq * 2.f, z, __fmul_rn(g_q, fmaf(-2.f, z, 1.f))));
    const float g_zr = (zr > 0.f && zr < 1.f) ? g_z : 0.f;
    gx = g_zr / w;
    g_x0 = -g_zr / w;
    float g_w = -g_zr * zr / w - g_s * s / w;
    g_h += g_s / w;
    g_x1 = g_w;
    g_x0 -= g_w;
    g_y1 = g_h;
    g_y0 = gy - g_h;
  }
  // interior knot k (1 <= k <= K-1) is rmin + sum of the bins before it: bin i
  // collects the gradients of the bin's two knots that lie beyond i
  const float ax1 = kb + 1 <= K - 1 ? g_x1 : 0.f, ay1 = kb + 1 <= K - 1 ? g_y1 : 0.f;
  const float axs = kb >= 1 ? ax1 + g_x0 : ax1, ays = kb >= 1 ? ay1 + g_y0 : ay1;
  const float gw_eq = __fmul_rn(ax1, scale), gh_eq = __fmul_rn(ay1, scale);
  const float gw_lt = __fmul_rn(axs, scale), gh_lt = __fmul_rn(ays, scale);
  float dw = 0.f, dh = 0.f;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    dw = fmaf(pw[i], i < kb ? gw_lt : i == kb ? gw_eq : 0.f, dw);
    dh = fmaf(ph[i], i < kb ? gh_lt : i == kb ? gh_eq : 0.f, dh);
  }
#pragma unroll
  for (int i = 0; i < K; ++i) {
    put(i, pw[i] * __fsub_rn(i < kb ? gw_lt : i == kb ? gw_eq : 0.f, dw));
    put(K + i, ph[i] * __fsub_rn(i < kb ? gh_lt : i == kb ? gh_eq : 0.f, dh));
  }
  // slopes: d_k = softplus(raw + off) + min_slope -> sigmoid
  const float s0 = g_d0 * (1.f / (1.f + expf(-(r0 + c.slope_offset))));
  const float s1 = g_d1 * (1.f / (1.f + expf(-(r1 + c.slope_offset))));
#pragma unroll
  for (int k = 0; k <= K; ++k) put(2 * K + k, k == k0 ? s0 : k == k1 ? s1 : 0.f);
  return gx;
}

// ---------------------------------------------------------------- inference, one bin
// Inference-only spline for the BF16 path: the same function as rqs_apply, with
// only the bin that holds v built. Both softmax
// normalisers are still needed (every knot depends on them), the knot
// positions are running sums whose last value at or below v picks the bin
// (identical to the one-hot selection: knots increase, so exactly one k has
// knot_k <= v < knot_{k+1}), and only that bin's two slopes go through the
// softplus. Exponentials, logarithms and divisions use the fast hardware
// approximations; with bf16 conditioner weights their error is far below the
// inputs' own rounding. raw: the 3K+1 conditioner outputs with bias added.
// log(1 + e) with e = exp(-|a|) <= 1 as __logf(1 + e): where 1 + e rounds
// to 1 the error is at most e < 2^-24 in absolute terms, far below the
// minimum knot slope (1e-4) the result is added to
__device__ __forceinline__ float softplus_fast(float a) {
  return fmaxf(a, 0.f) + __logf(1.f + __expf(-fabsf(a)));
}

// 2^x on the SFU (ex2.approx.ftz.f32); softmax arguments are <= 0 after the
// max subtraction, so the approximation's relative error bounds the result
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed FP32 pairs (f32x2: two lanes of a 64-bit register pair per
// instruction) and the three-input maximum, both sm_100-family instructions.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// a[i] += b[i] for i < N, adjacent pairs as one f32x2 add
template <int N>
__device__ __forceinline__ void add_f2(float* a, const float* b) {
#pragma unroll
  for (int i = 0; i + 1 < N; i += 2) f2_unpack(f2_add(f2_pack(a[i], a[i + 1]), f2_pack(b[i], b[i + 1])), a[i], a[i + 1]);
  if (N & 1) a[N - 1] += b[N - 1];
}

// Unnormalised softmax weights of the K bin widths and K bin heights,
// ew[k] = e^(raw[k] - max) as one FFMA + ex2 each, and their sums. The
// FFMAs and the sums run on adjacent pairs as f32x2 (the sums as two
// interleaved partial sums, added at the end).
template <int K>
__device__ __forceinline__ void softmax_weights(const float (&raw)[3 * K + 1], float (&ew)[K], float (&eh)[K],
                                                float& sw, float& sh) {
  constexpr float kLog2e = 1.4426950408889634f;
  float mw = raw[0], mh = raw[K];
#pragma unroll
  for (int k = 1; k < K; k += 2) {
    if (k + 1 < K) {
      mw = fmax3(mw, raw[k], raw[k + 1]);
      mh = fmax3(mh, raw[K + k], raw[K + k + 1]);
    } else {
      mw = fmaxf(mw, raw[k]);
      mh = fmaxf(mh, raw[K + k]);
    }
  }
  const float nmw = -mw * kLog2e, nmh = -mh * kLog2e;
  const uint64_t l2 = f2_pack(kLog2e, kLog2e), nw2 = f2_pack(nmw, nmw), nh2 = f2_pack(nmh, nmh);
  uint64_t sw2 = f2_pack(0.f, 0.f), sh2 = sw2;
#pragma unroll
  for (int k = 0; k + 1 < K; k += 2) {
    float a0, a1, b0, b1;
    f2_unpack(f2_fma(f2_pack(raw[k], raw[k + 1]), l2, nw2), a0, a1);
    f2_unpack(f2_fma(f2_pack(raw[K + k], raw[K + k + 1]), l2, nh2), b0, b1);
    ew[k] = ex2_approx(a0);
    ew[k + 1] = ex2_approx(a1);
    eh[k] = ex2_approx(b0);
    eh[k + 1] = ex2_approx(b1);
    sw2 = f2_add(sw2, f2_pack(ew[k], ew[k + 1]));
    sh2 = f2_add(sh2, f2_pack(eh[k], eh[k + 1]));
  }
  float a, b;
  f2_unpack(sw2, a, b);
  sw = a + b;
  f2_unpack(sh2, a, b);
  sh = a + b;
  if (K & 1) {
    ew[K - 1] = ex2_approx(fmaf(raw[K - 1], kLog2e, nmw));
    eh[K - 1] = ex2_approx(fmaf(raw[2 * K - 1], kLog2e, nmh));
    sw += ew[K - 1];
    sh += eh[K - 1];
  }
}

// The spline of the bin that holds v only, for the fused tensor-core
// epilogue (same function as rqs_apply up to rounding):
// unnormalised softmax weights (softmax_weights), the bin
// found by comparing v with the running knots while carrying only what the
// bin needs (cumulative sums before it, its own weights, its two slope
// parameters), and one log for the log-determinant.
template <int K, bool INV>
__device__ __forceinline__ void rqs_apply_fast(const float (&raw)[3 * K + 1], float v, const SplineCfg& c, float& out,
                                               float& ld) {
  float ew[K], eh[K], sw, sh;
  softmax_weights<K>(raw, ew, eh, sw, sh);
  const float scale = (c.rmax - c.rmin) - (float)K * c.min_bin;
  const float isw = __fdividef(1.f, sw), ish = __fdividef(1.f, sh), iscale = __fdividef(1.f, scale);
  const float fw = scale * isw, fh = scale * ish;   // knot spacing per unit of softmax weight
  // knot k = rmin + f * (sum_{j<k} e_j + k * min_bin / f) = rmin + f * (sum_{j<k} e'_j)
  // with e'_j = e_j + min_bin / f: the bin is found by comparing the running
  // sums of e' with (v - rmin) / f (no per-knot multiply), its left knots are
  // rmin + f * (the sums before it) and its width and height f * e'_bin. Bin 0
  // by default (also covers v below the range).
  const float dw = c.min_bin * sw * iscale, dh = c.min_bin * sh * iscale;
  float ewp[K], ehp[K];
#pragma unroll
  for (int k = 0; k + 1 < K; k += 2) {
    f2_unpack(f2_add(f2_pack(ew[k], ew[k + 1]), f2_pack(dw, dw)), ewp[k], ewp[k + 1]);
    f2_unpack(f2_add(f2_pack(eh[k], eh[k + 1]), f2_pack(dh, dh)), ehp[k], ehp[k + 1]);
  }
  if (K & 1) {
    ewp[K - 1] = ew[K - 1] + dw;
    ehp[K - 1] = eh[K - 1] + dh;
  }
  const float a = (v - c.rmin) * (INV ? sh : sw) * iscale;
  float cw = 0.f, ch = 0.f, bw = 0.f, bh = 0.f, ebw = ewp[0], ebh = ehp[0];
  float r0 = raw[2 * K], r1 = raw[2 * K + 1];
  bool last = false;   // the bin is the last one, whose right knot is exactly rmax
#pragma unroll
  for (int k = 1; k < K; ++k) {
    cw += ewp[k - 1];
    ch += ehp[k - 1];
    const bool in = (INV ? ch : cw) <= a;
    if (in) {
      bw = cw; bh = ch; ebw = ewp[k]; ebh = ehp[k];
      r0 = raw[2 * K + k];
      r1 = raw[2 * K + k + 1];
    }
    if (k == K - 1) last = in;
  }
  const float x0 = fmaf(bw, fw, c.rmin);
  const float y0 = fmaf(bh, fh, c.rmin);
  const float w = last ? c.rmax - x0 : ebw * fw;
  const float h = last ? c.rmax - y0 : ebh * fh;
  const float d0 = softplus_fast(r0 + c.slope_offset) + c.min_slope;
  const float d1 = softplus_fast(r1 + c.slope_offset) + c.min_slope;
  const float s = __fdividef(h, w);
  const float st = d1 + d0 - 2.f * s;
  float z;
  if (!INV) {
    z = fminf(fmaxf(__fdividef(v - x0, w), 0.f), 1.f);
  } else {
    const float ww = fminf(fmaxf(__fdividef(v - y0, h), 0.f), 1.f);
    const float cq = -s * ww;
    const float bq = d0 - st * ww;
    const float aq = s - bq;
    const float disc = bq * bq - 4.f * aq * cq;
    // the hardware square-root approximation (one instruction), like the
    // other fast approximations of this path
    float sqd = 0.f;
    if (disc > 0.f) asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sqd) : "f"(disc));
    const float num = (bq >= 0.f) ? 2.f * cq : -bq + sqd;
    const float dnm = (bq >= 0.f) ? -bq - sqd : 2.f * aq;
    z = fminf(fmaxf(__fdividef(num, dnm), 0.f), 1.f);
  }
  const float sq = z * z, q = z - sq, om = 1.f - z;
  const float den = s + st * q;
  const float A = d1 * sq + 2.f * s * q + d0 * om * om;
  // log-det 2 log s + log A - 2 log den as one log; log d0 / log d1 in the tails
  float arg = __fdividef(s * s * A, den * den);
  if (!INV) {
    out = y0 + __fdividef(h * (s * sq + d0 * q), den);
    if (v <= c.rmin) { out = (v - c.rmin) * d0 + c.rmin; arg = d0; }
    if (v >= c.rmax) { out = (v - c.rmax) * d1 + c.rmax; arg = d1; }
    ld = __logf(arg);
  } else {
    out = w * z + x0;
    if (v <= c.rmin) { out = __fdividef(v - c.rmin, d0) + c.rmin; arg = d0; }
    if (v >= c.rmax) { out = __fdividef(v - c.rmax, d1) + c.rmax; arg = d1; }
    ld = -__logf(arg);
  }
}

// Adjoint of rqs_apply_fast<K, false> for the BF16 training path: given
// gy = dL/dy and gl = dL/dlogdet, returns dL/dx and writes dL/draw[0..3K] as
// bf16 to out. Same derivative as rqs_adjoint, organised around the one
// bin that holds x: only its two knots carry gradient into the cumulative
// widths/heights (so dL/dw_i is a two-term prefix rule) and only its two
// slopes go through the softplus derivative; the rest of the slope
// gradients are exactly zero.
template <int K>
__device__ __forceinline__ float rqs_fwd_adjoint_fast(const float (&raw)[3 * K + 1], float x, float gy, float gl,
                                                      const SplineCfg& c, uint16_t* __restrict__ out) {
  float pw[K], ph[K], sw, sh;
  softmax_weights<K>(raw, pw, ph, sw, sh);
  const float iw = __fdividef(1.f, sw), ih = __fdividef(1.f, sh);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    pw[k] *= iw;
    ph[k] *= ih;
  }
  const float scale = (c.rmax - c.rmin) - (float)K * c.min_bin;
  // the bin: cumulative probabilities before it and its own (see rqs_apply_fast)
  float cpw = 0.f, cph = 0.f, bwn = 0.f, bhn = 0.f, ebw = pw[0], ebh = ph[0];
  float r0 = raw[2 * K], r1 = raw[2 * K + 1];
  int kb = 0;
#pragma unroll
  for (int k = 1; k < K; ++k) {
    cpw += pw[k - 1];
    cph += ph[k - 1];
    if (x >= fmaf(cpw, scale, fmaf((float)k, c.min_bin, c.rmin))) {
      bwn = cpw; bhn = cph; ebw = pw[k]; ebh = ph[k]; kb = k;
      r0 = raw[2 * K + k];
      r1 = raw[2 * K + k + 1];
    }
  }
  const bool last = kb == K - 1;   // the last knot is exactly rmax
  const float x0 = fmaf(bwn, scale, fmaf((float)kb, c.min_bin, c.rmin));
  const float y0 = fmaf(bhn, scale, fmaf((float)kb, c.min_bin, c.rmin));
  const float x1 = last ? c.rmax : x0 + fmaf(ebw, scale, c.min_bin);
  const float y1 = last ? c.rmax : y0 + fmaf(ebh, scale, c.min_bin);
  const float a0 = r0 + c.slope_offset, a1 = r1 + c.slope_offset;
  const float d0 = softplus_fast(a0) + c.min_slope, d1 = softplus_fast(a1) + c.min_slope;
  float gx, g_x0 = 0.f, g_x1 = 0.f, g_y0 = 0.f, g_y1 = 0.f, g_d0 = 0.f, g_d1 = 0.f;
  if (x <= c.rmin) {
    gx = gy * d0;
    g_d0 = gy * (x - c.rmin) + __fdividef(gl, d0);
  } else if (x >= c.rmax) {
    gx = gy * d1;
    g_d1 = gy * (x - c.rmax) + __fdividef(gl, d1);
  } else {
    const float w = x1 - x0, h = y1 - y0;
    const float iwd = __fdividef(1.f, w);
    const float s = h * iwd;
    const float zr = (x - x0) * iwd;
    const float z = fminf(fmaxf(zr, 0.f), 1.f);
    const float sq = z * z, q = z - sq, om = 1.f - z, sq1 = om * om;
    const float st = d1 + d0 - 2.f * s;
    const float num = h * (s * sq + d0 * q);
    const float den = s + st * q;
    const float A = d1 * sq + 2.f * s * q + d0 * sq1;
    const float iden = __fdividef(1.f, den);
    // y = y0 + num/den ; ld = 2 log s + log A - 2 log den
    const float g_num = gy * iden;
    const float g_den = -(gy * num * iden + 2.f * gl) * iden;
    const float g_A = __fdividef(gl, A);
    float g_s = __fdividef(2.f * gl, s);
    float g_h = g_num * (s * sq + d0 * q);
    g_s += g_num * h * sq;
    float g_sq = g_num * h * s;
    g_d0 = g_num * h * q;
    float g_q = g_num * h * d0;
    g_s += g_den * (1.f - 2.f * q);
    g_d1 = g_den * q;
    g_d0 += g_den * q;
    g_q += g_den * st;
    g_d1 += g_A * sq;
    g_sq += g_A * d1;
    g_s += g_A * 2.f * q;
    g_q += g_A * 2.f * s;
    g_d0 += g_A * sq1;
    float g_z = -g_A * d0 * 2.f * om;
    g_z += g_q * (1.f - 2.f * z) + g_sq * 2.f * z;
    const float g_zr = (zr > 0.f && zr < 1.f) ? g_z : 0.f;
    gx = g_zr * iwd;
    const float g_w = -(g_zr * zr + g_s * s) * iwd;
    g_h += g_s * iwd;
    g_x0 = -g_zr * iwd - g_w;
    g_x1 = g_w;
    g_y1 = g_h;
    g_y0 = gy - g_h;
  }
  // interior knot k (1 <= k <= K-1) is rmin + sum_{i<k} width_i: dL/dwidth_i
  // collects the gradients of the bin's two knots that lie beyond i, i.e.
  // scale (ax0 + ax1) for i < kb, scale ax1 for i = kb, 0 beyond; the softmax
  // adjoint's sum_j p_j g_j is then closed-form in the bin's sums
  const float ax0 = (kb >= 1) ? g_x0 : 0.f, ax1 = (kb + 1 <= K - 1) ? g_x1 : 0.f;
  const float ay0 = (kb >= 1) ? g_y0 : 0.f, ay1 = (kb + 1 <= K - 1) ? g_y1 : 0.f;
  const float gw_lt = scale * (ax0 + ax1), gw_eq = scale * ax1;
  const float gh_lt = scale * (ay0 + ay1), gh_eq = scale * ay1;
  const float dw = gw_lt * bwn + gw_eq * ebw, dh = gh_lt * bhn + gh_eq * ebh;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const float gwi = (i < kb) ? gw_lt : ((i == kb) ? gw_eq : 0.f);
    const float ghi = (i < kb) ? gh_lt : ((i == kb) ? gh_eq : 0.f);
    out[i] = __bfloat16_as_ushort(__float2bfloat16_rn(pw[i] * (gwi - dw)));
    out[K + i] = __bfloat16_as_ushort(__float2bfloat16_rn(ph[i] * (ghi - dh)));
  }
  // slopes: d = softplus(raw + offset) + min_slope, d' = sigmoid(raw + offset)
  const float gs0 = g_d0 * __fdividef(1.f, 1.f + __expf(-a0));
  const float gs1 = g_d1 * __fdividef(1.f, 1.f + __expf(-a1));
#pragma unroll
  for (int k = 0; k <= K; ++k) {
    const float v = (k == kb ? gs0 : 0.f) + (k == kb + 1 ? gs1 : 0.f);
    out[2 * K + k] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
  }
  return gx;
}

}  // namespace fmc
