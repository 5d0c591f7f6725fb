// gemm_f32.cuh -- FP32 SIMT GEMMs of the RealNVP flow.
//
//   k_gemm_f32    C[m, n] = epi(sum_k A[m, k] B[n, k]), both operands K-major
//   k_kouter_f32  sums over row slices of G[row, m] X[row, n] (weight gradients)
//
// Both stage 16 inputs at a time through shared memory with cp.async (two
// stages in flight) and multiply packed pairs (fma.rn.f32x2), which reach 72
// TFLOP/s on GB300 where plain FMAs stop at 52 (register ports). The K-major GEMM
// pairs adjacent inputs -- even and odd inputs summed apart, added at the end --
// so neither operand has to be duplicated (the gradient's products; the forward's
// are plain FMAs in input order, see gemm_f32); the outer product pairs adjacent m.
// A 16-byte shared-memory load costs two cycles when each quarter warp reads at
// most two addresses and four otherwise, so the row operand is the one that
// quarters of a warp share: 8 x 8 outputs per thread keep the loads at three
// quarters of the FMA time, 8 x 4 (outputs of at most 32) at its whole.
#pragma once
#include <type_traits>
#include "flow.cuh"

namespace fmc {

constexpr int kG32BK = 16, kG32Pitch = 20, kG32Stages = 3;

enum G32Epi : int {
  G32_BIAS = 0,       // C = AB + bias
  G32_BIAS_RELU = 1,  // C = max(AB + bias, 0)
  G32_DRELU = 2,      // C = AB where aux > 0, else 0
  G32_ADD_MASKED = 3  // C += AB * bias[n]   (bias: the column mask)
};

// one problem of a launch (blockIdx.z)
struct G32Problem {
  const float* A;
  const float* B;
  const float* bias;
  const float* aux;
  float* C;
};
struct G32Args {
  G32Problem p[2];
  int64_t M, lda, ldb, ldaux, ldc;
  int N, K;
};

// 4 RM WR rows x 8 TN columns per CTA; WR warps of 4 x 8 lanes with RM x TN outputs
// per thread, times WK groups of warps that take every WK-th 16-input chunk
// (outputs too few to fill the SMs: the groups' sums are added through shared
// memory in order). The tile leaves through shared memory as whole rows.
template <int WR, int TN, int WK, int EPI, bool SEQ, int RM = 8>
__global__ void __launch_bounds__(32 * WR * WK, TN == 4 ? 2 * RM / (WR * WK) : 1) k_gemm_f32(const __grid_constant__ G32Args a) {
  constexpr int NT = 32 * WR * WK, BM = 4 * RM * WR, BN = 8 * TN, ROWS = BM + BN;
  constexpr int STAGE = WK * ROWS * kG32Pitch, LDT = BN + 8, BKS = WK * kG32BK;
  extern __shared__ __align__(16) float sm[];
  const G32Problem& p = a.p[blockIdx.z];
  const int tid = threadIdx.x, lane = tid & 31, wid = (tid >> 5) % WR, grp = (tid >> 5) / WR;
  const int64_t m0 = (int64_t)blockIdx.y * BM;
  const int n0 = blockIdx.x * BN;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
  // 16-, 8- or 4-byte copies, as an operand's rows are aligned
  auto width = [&](const float* q, int64_t ld) {
    const uintptr_t al = (uintptr_t)q | (uintptr_t)(4 * (ld | a.K));
    return (al & 15) == 0 ? 4 : (al & 7) == 0 ? 2 : 1;
  };
  const int wa = width(p.A, a.lda), wb = width(p.B, a.ldb);
  // `rows` rows of an operand from row r0 of `limit`; rows past the limit and
  // inputs past K, up to a multiple of four, are copied as zeros
  auto copy_w = [&](auto floats, auto rows, const float* src, int64_t ld, int64_t r0, int64_t limit, int k0, uint32_t dst) {
    constexpr int PER = decltype(floats)::value, CH = kG32BK / PER, R = decltype(rows)::value;
#pragma unroll 4
    for (int e = tid; e < WK * R * CH; e += NT) {
      const int q = e % CH, rr = e / CH, r = rr % R, kc = rr / R;
      const int k = k0 + kc * kG32BK + PER * q;
      if (k >= ((a.K + 3) & ~3)) continue;
      const bool in = k < a.K && r0 + r < limit;
      const float* g = in ? src + (r0 + r) * ld + k : src;
      const uint32_t d = dst + 4 * ((kc * ROWS + r) * kG32Pitch + PER * q);
      if (PER == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g), "r"(in ? 16 : 0));
      else if (PER == 2)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(g), "r"(in ? 8 : 0));
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(g), "r"(in ? 4 : 0));
    }
  };
  auto copy = [&](int w, auto rows, const float* src, int64_t ld, int64_t r0, int64_t limit, int k0, uint32_t dst) {
    if (w == 4) copy_w(IntC<4>{}, rows, src, ld, r0, limit, k0, dst);
    else if (w == 2) copy_w(IntC<2>{}, rows, src, ld, r0, limit, k0, dst);
    else copy_w(IntC<1>{}, rows, src, ld, r0, limit, k0, dst);
  };
  auto issue = [&](int k0, int slot) {
    if (k0 < a.K) {
      const uint32_t dst = sbase + slot * (4 * STAGE);
      copy(wa, IntC<BM>{}, p.A, a.lda, m0, a.M, k0, dst);
      copy(wb, IntC<BN>{}, p.B, a.ldb, n0, a.N, k0, dst + 4 * BM * kG32Pitch);
    }
    asm volatile("cp.async.commit_group;");
  };
  const int r0 = wid * (4 * RM) + (lane >> 3), c0 = lane & 7;   // rows r0 + 4 i, columns c0 + 8 j
  using Acc = std::conditional_t<SEQ, float, uint64_t>;
  Acc acc[RM][TN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = Acc(0);
#pragma unroll
  for (int q = 0; q < kG32Stages - 1; ++q) issue(q * BKS, q);
  int slot = 0;
  for (int k0 = 0; k0 < a.K; k0 += BKS) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kG32Stages - 2) : "memory");
    __syncthreads();
    issue(k0 + (kG32Stages - 1) * BKS, slot == 0 ? kG32Stages - 1 : slot - 1);
    if (k0 + grp * kG32BK < a.K) {
      const float* As = sm + slot * STAGE + (grp * ROWS + r0) * kG32Pitch;
      const float* Bs = sm + slot * STAGE + (grp * ROWS + BM + c0) * kG32Pitch;
#pragma unroll
      for (int k = 0; k < kG32BK; k += 4) {
        if (k0 + grp * kG32BK + k >= a.K) break;
        if constexpr (SEQ) {
          float4 b[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(Bs + 8 * j * kG32Pitch + k);
#pragma unroll
          for (int i = 0; i < RM; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(As + 4 * i * kG32Pitch + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(v.x, b[j].x, acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(v.y, b[j].y, acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(v.z, b[j].z, acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(v.w, b[j].w, acc[i][j]);
          }
        } else {
          ulonglong2 b[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(Bs + 8 * j * kG32Pitch + k);
#pragma unroll
          for (int i = 0; i < RM; ++i) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(As + 4 * i * kG32Pitch + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
              acc[i][j] = f2_fma(v.x, b[j].x, acc[i][j]);
              acc[i][j] = f2_fma(v.y, b[j].y, acc[i][j]);
            }
          }
        }
      }
    }
    slot = slot + 1 == kG32Stages ? 0 : slot + 1;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      float v;
      if constexpr (SEQ) {
        v = acc[i][j];
      } else {
        float lo, hi;
        f2_unpack(acc[i][j], lo, hi);
        v = lo + hi;
      }
      sm[(grp * BM + r0 + 4 * i) * LDT + c0 + 8 * j] = v;
    }
  __syncthreads();
  const bool vout = (a.ldc & 3) == 0 && (a.N & 3) == 0 && ((uintptr_t)p.C & 15) == 0 &&
                    (EPI != G32_DRELU || ((a.ldaux & 3) == 0 && ((uintptr_t)p.aux & 15) == 0));
  auto one = [&](float v, float aux, int n, float c) {
    if (EPI == G32_BIAS) return v + __ldg(p.bias + n);
    if (EPI == G32_BIAS_RELU) return fmaxf(v + __ldg(p.bias + n), 0.f);
    if (EPI == G32_DRELU) return aux > 0.f ? v : 0.f;
    return fmaf(v, __ldg(p.bias + n), c);
  };
  if (vout) {
#pragma unroll 4
    for (int e = tid; e < BM * BN / 4; e += NT) {
      const int r = e / (BN / 4), c = 4 * (e % (BN / 4)), n = n0 + c;
      const int64_t m = m0 + r;
      if (m >= a.M || n >= a.N) continue;
      float4 v = *reinterpret_cast<const float4*>(sm + r * LDT + c);
#pragma unroll
      for (int g = 1; g < WK; ++g) {
        const float4 t = *reinterpret_cast<const float4*>(sm + (g * BM + r) * LDT + c);
        v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
      }
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), o = x;
      if (EPI == G32_DRELU) x = *reinterpret_cast<const float4*>(p.aux + m * a.ldaux + n);
      float4* dst = reinterpret_cast<float4*>(p.C + m * a.ldc + n);
      if (EPI == G32_ADD_MASKED) o = *dst;
      *dst = make_float4(one(v.x, x.x, n, o.x), one(v.y, x.y, n + 1, o.y), one(v.z, x.z, n + 2, o.z),
                         one(v.w, x.w, n + 3, o.w));
    }
  } else {
    for (int e = tid; e < BM * BN; e += NT) {
      const int r = e / BN, c = e % BN, n = n0 + c;
      const int64_t m = m0 + r;
      if (m >= a.M || n >= a.N) continue;
      float v = sm[r * LDT + c];
#pragma unroll
      for (int g = 1; g < WK; ++g) v += sm[(g * BM + r) * LDT + c];
      float* dst = p.C + m * a.ldc + n;
      *dst = one(v, EPI == G32_DRELU ? p.aux[m * a.ldaux + n] : 0.f, n, EPI == G32_ADD_MASKED ? *dst : 0.f);
    }
  }
}

// `count` problems (1 or 2) of one shape in a launch: 128 x 64 tiles of four
// warps; 128 x 32 for few inputs (a tile is then mostly latency and output
// traffic: half the registers, twice the CTAs per SM; [16384 x 32] x [32 x 256],
// two with relu masks, 51 -> 37 us); for outputs of at most 32 columns, and where
// the wide tiles would leave SMs idle, 64 x 32 of two warps times four input
// groups ([16384 x 512] x [512 x 32] 32 -> 25 us)
//
// The forward epilogues (SEQ) add an output's products one by one in the order
// of the inputs, so that the bits do not depend on the tile: a row's results are the
// same in a call of one row and of a million, the loss is that of log_prob,
// and the relu derivative of a kept activation, which jumps where its input is 0,
// is that of the forward. The gradient's products, summed over the batch anyway,
// take packed sums of even and odd inputs, and of input groups.
template <int EPI>
inline int gemm_f32(cudaStream_t st, const G32Args& a, int count) {
  constexpr bool SEQ = EPI == G32_BIAS || EPI == G32_BIAS_RELU;
  if (a.M <= 0 || a.N <= 0) return FMC_OK;
  auto go = [&](auto kern, int bm, int bn, int wk, int threads) -> int {
    const int smem = kG32Stages * wk * (bm + bn) * kG32Pitch * 4;
    FMC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    // tall problems in launches of at most 65,535 row tiles
    G32Args b = a;
    const int64_t step = 65535ll * bm;
    for (int64_t m = 0; m < a.M; m += step) {
      b.M = a.M - m < step ? a.M - m : step;
      for (int z = 0; z < count; ++z) {
        b.p[z].A = a.p[z].A + m * a.lda;
        b.p[z].C = a.p[z].C + m * a.ldc;
        b.p[z].aux = a.p[z].aux ? a.p[z].aux + m * a.ldaux : nullptr;
      }
      kern<<<dim3((unsigned)((a.N + bn - 1) / bn), (unsigned)((b.M + bm - 1) / bm), (unsigned)count), threads, smem, st>>>(b);
      FMC_LAUNCH_CHECK();
    }
    return FMC_OK;
  };
  const int64_t wide = (a.M + 127) / 128 * ((a.N + 63) / 64) * count;
  if (a.N <= 32 || wide < sm_count()) {
    if constexpr (SEQ) {
      // tiles that leave SMs idle: a quarter of the outputs per thread on four times
      // the warps, where packed sums would split the inputs (log_prob of 100 rows, 32-D,
      // 8 layers, H = 256: 226 -> 177 us, 500 rows of 64-D, 4 layers, H = 64: 94 -> 78; up to
      // two tiles per SM it was 0.9 to 1.07 of the time)
      if ((a.M + 63) / 64 * ((a.N + 31) / 32) * count <= sm_count())
        return go(k_gemm_f32<8, 4, 1, EPI, SEQ, 2>, 64, 32, 1, 256);
      return go(k_gemm_f32<2, 4, 1, EPI, SEQ>, 64, 32, 1, 64);
    } else {
      return go(k_gemm_f32<2, 4, 4, EPI, SEQ>, 64, 32, 4, 256);
    }
  }
  if (a.K <= 64) return go(k_gemm_f32<4, 4, 1, EPI, SEQ>, 128, 32, 1, 128);
  return go(k_gemm_f32<4, 8, 1, EPI, SEQ>, 128, 64, 1, 128);
}

// ------------------------------------------------------------------ weight gradients
// one weight matrix of every layer: layer l at G + l layer_g, X + l layer_x
struct K32Problem {
  const float* G;   // [rows, ldg]
  const float* X;   // [rows, ldx]
  int64_t layer_g, layer_x, ldg, ldx;
  int M, N;
  int64_t off, sm, sn;   // element (m, n) at off + m sm + n sn of the layer's parameters
};
struct K32Args {
  K32Problem p[3];
  int n_problems;                 // blockIdx.z = layer * n_problems + problem
  int64_t rows, rows_per_slice;   // slices: blockIdx.y
  int64_t per_layer, n_params;
  float* part;                    // [slices][n_params]
};

constexpr int kK32N = 32, kK32M = 256, kK32Threads = 128;
constexpr int kK32StageFloats = kG32BK * (kK32M + kK32N);

// 256 x 32 tiles, four warps of 64 x 32, 16 x 4 outputs per thread
__global__ void __launch_bounds__(kK32Threads, 2) k_kouter_f32(const __grid_constant__ K32Args a) {
  extern __shared__ __align__(16) float sm[];
  const K32Problem& p = a.p[blockIdx.z % a.n_problems];
  const int64_t layer = blockIdx.z / a.n_problems;
  const float* Gl = p.G + layer * p.layer_g;
  const float* Xl = p.X + layer * p.layer_x;
  const int tn = (p.N + kK32N - 1) / kK32N, tm = (p.M + kK32M - 1) / kK32M;
  if ((int)blockIdx.x >= tn * tm) return;
  const int m0 = (int)blockIdx.x / tn * kK32M, n0 = (int)blockIdx.x % tn * kK32N;
  const int64_t k_begin = (int64_t)blockIdx.y * a.rows_per_slice;
  const int64_t k_end = k_begin + a.rows_per_slice < a.rows ? k_begin + a.rows_per_slice : a.rows;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
  auto width = [](const float* q, int64_t ld, int cols) {
    const uintptr_t al = (uintptr_t)q | (uintptr_t)(4 * (ld | cols));
    return (al & 15) == 0 ? 4 : (al & 7) == 0 ? 2 : 1;
  };
  const int vg = width(Gl, p.ldg, p.M), vx = width(Xl, p.ldx, p.N);
  // rows past the slice and columns past M or N are copied as zeros
  auto copy_w = [&](auto floats, auto cols_s, const float* src, int64_t ld, int c0, int cols, int64_t k, uint32_t dst) {
    constexpr int PER = decltype(floats)::value, W = decltype(cols_s)::value;
#pragma unroll 4
    for (int e = tid; e < kG32BK * W / PER; e += kK32Threads) {
      const int r = e / (W / PER), c = PER * (e % (W / PER));
      const bool in = k + r < k_end && c0 + c < cols;
      const float* q = in ? src + (k + r) * ld + c0 + c : src;
      const uint32_t d = dst + 4 * (r * W + c);
      if (PER == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(q), "r"(in ? 16 : 0));
      else if (PER == 2)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(q), "r"(in ? 8 : 0));
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(q), "r"(in ? 4 : 0));
    }
  };
  auto copy = [&](auto cols_s, const float* src, int64_t ld, int c0, int cols, int64_t k, uint32_t dst, int v) {
    if (v == 4) copy_w(IntC<4>{}, cols_s, src, ld, c0, cols, k, dst);
    else if (v == 2) copy_w(IntC<2>{}, cols_s, src, ld, c0, cols, k, dst);
    else copy_w(IntC<1>{}, cols_s, src, ld, c0, cols, k, dst);
  };
  auto issue = [&](int64_t k, int slot) {
    if (k < k_end) {
      const uint32_t dst = sbase + slot * (4 * kK32StageFloats);
      copy(IntC<kK32M>{}, Gl, p.ldg, m0, p.M, k, dst, vg);
      copy(IntC<kK32N>{}, Xl, p.ldx, n0, p.N, k, dst + 4 * kG32BK * kK32M, vx);
    }
    asm volatile("cp.async.commit_group;");
  };
  const int mr = wid * 64 + (lane >> 3) * 4, nr = (lane & 7) * 4;   // outputs mr + 16 i + 0..3, nr + 0..3
  uint64_t acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0ull;
  const bool on = m0 + wid * 64 < p.M;
#pragma unroll
  for (int q = 0; q < kG32Stages - 1; ++q) issue(k_begin + q * kG32BK, q);
  int slot = 0;
  for (int64_t k = k_begin; k < k_end; k += kG32BK) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kG32Stages - 2) : "memory");
    __syncthreads();
    issue(k + (kG32Stages - 1) * kG32BK, slot == 0 ? kG32Stages - 1 : slot - 1);
    if (on) {
      const float* Gs = sm + slot * kK32StageFloats + mr;
      const float* Xs = sm + slot * kK32StageFloats + kG32BK * kK32M + nr;
#pragma unroll
      for (int kk = 0; kk < kG32BK; ++kk) {
        const float4 x = *reinterpret_cast<const float4*>(Xs + kk * kK32N);
        const uint64_t b[4] = {f2_pack(x.x, x.x), f2_pack(x.y, x.y), f2_pack(x.z, x.z), f2_pack(x.w, x.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Gs + kk * kK32M + 16 * i);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[i][j][0] = f2_fma(v.x, b[j], acc[i][j][0]);
            acc[i][j][1] = f2_fma(v.y, b[j], acc[i][j][1]);
          }
        }
      }
    }
    slot = slot + 1 == kG32Stages ? 0 : slot + 1;
  }
  float* out = a.part + (int64_t)blockIdx.y * a.n_params + layer * a.per_layer + p.off;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v[4];
      f2_unpack(acc[i][j][0], v[0], v[1]);
      f2_unpack(acc[i][j][1], v[2], v[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = m0 + mr + 16 * i + e, n = n0 + nr + j;
        if (m < p.M && n < p.N) out[m * p.sm + n * p.sn] = v[e];
      }
    }
}

}  // namespace fmc
