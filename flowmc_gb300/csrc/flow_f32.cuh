// flow_f32.cuh -- building blocks of the fused FP32 flow kernels (flow_f32.cu):
// a CTA keeps a tile of R rows in shared memory and runs the conditioner's
// Linears and the splines of every layer on it.
//
// The products are SIMT: C[row, n] = sum_k A[row, k] W[n, k], one FMA chain in k
// order per element (the bits of a plain SIMT GEMM). A (activations) lies
// input-major in shared memory ([k][row]), W streams from L2 in stages of 128
// outputs x 16 inputs that run on across Linears and layers. FMAs are packed
// pairs over two adjacent rows (fma.rn.f32x2, the weight in both halves), which
// leaves issue slots for the shared-memory loads and the moves that pair up the
// weights. A shared-memory load returns 128 bytes per cycle whatever it
// broadcasts, against 128 FMAs per cycle, so an 8 x 4 tile per thread is held to
// two thirds of the FMA rate by its loads; 64-row tiles therefore take 8 x 8
// per thread on four warps, two CTAs per SM (one's splines beside the other's
// products). Lanes are 4 row groups x 8 outputs; a thread takes four consecutive
// rows per 16 and every eighth output, so each 16-byte load or store of a warp
// is free of bank conflicts (pitches of 20 floats for W, R + 4 for A).
#pragma once
#include "flow.cuh"

namespace fmc {

constexpr int kFlowCols = 128;                  // outputs per product tile
constexpr int kFlowBK = 16;                     // inputs per stage
constexpr int kFlowPitch = kFlowBK + 4;
constexpr int kFlowStageFloats = kFlowCols * kFlowPitch;

// geometry of the packed parameters in closed form (layers alternate between
// two parities), small enough to be a kernel argument
struct FlowShape {
  int d, L, nh, K, P, dg;     // dg: coordinates per tile of the last Linear
  int H[FMC_MAX_HIDDEN];
  int64_t par_size[2];        // parameters of an even / odd layer
  SplineCfg cfg;
  __host__ __device__ int cpar(int l) const { return 1 - (l & 1); }
  __host__ __device__ int tpar(int l) const { return l & 1; }
  __host__ __device__ int nc(int l) const { return (d - cpar(l) + 1) / 2; }
  __host__ __device__ int nt(int l) const { return d - nc(l); }
  __host__ __device__ int in(int l, int i) const { return i == 0 ? nc(l) : H[i - 1]; }
  __host__ __device__ int out(int l, int i) const { return i == nh ? nt(l) * P : H[i]; }
  __host__ __device__ int64_t layer_off(int l) const {
    return (int64_t)(l / 2) * (par_size[0] + par_size[1]) + (l & 1) * par_size[0];
  }
  __host__ __device__ int64_t w_off(int l, int i) const {   // within the layer
    int64_t o = 2;
    for (int u = 0; u < i; ++u) o += (int64_t)out(l, u) * (in(l, u) + 1);
    return o;
  }
  // columns of a layer's saved activations: conditioning block, hidden
  // activations, conditioner outputs (act_col: first column of Linear i's
  // input; i = nh + 1: its outputs), and of its output gradients
  __host__ __device__ int act_col(int l, int i) const {
    int c = 0;
    for (int u = 0; u < i; ++u) c += in(l, u);
    return c;
  }
  __host__ __device__ int act_cols(int l) const { return act_col(l, nh + 1) + out(l, nh); }
  __host__ __device__ int64_t act_base(int l) const {   // columns before layer l
    return (int64_t)(l / 2) * (act_cols(0) + act_cols(1)) + (l & 1) * act_cols(0);
  }
  // padded columns of the Linears' output gradients (rows of round_up(out, 4)
  // floats): those before Linear i of layer l
  __host__ __device__ int gpad(int l, int i) const { return (out(l, i) + 3) & ~3; }
  __host__ __device__ int gcols(int l) const {
    int c = 0;
    for (int u = 0; u <= nh; ++u) c += gpad(l, u);
    return c;
  }
  __host__ __device__ int64_t gcol(int l, int i) const {
    int64_t c = (int64_t)(l / 2) * (gcols(0) + gcols(1)) + (l & 1) * gcols(0);
    for (int u = 0; u < i; ++u) c += gpad(l, u);
    return c;
  }
  // outputs per product tile of Linear i
  __host__ __device__ int tile_cols(int i) const { return i == nh ? dg * P : kFlowCols; }
};

inline FlowShape flow_shape(const FlowGeom& g) {
  FlowShape s{};
  s.d = g.d;
  s.L = g.L;
  s.nh = g.nh;
  s.K = g.K;
  s.P = g.P;
  s.dg = kFlowCols / g.P;
  for (int i = 0; i < FMC_MAX_HIDDEN; ++i) s.H[i] = g.H[i];
  for (int l = 0; l < 2; ++l) s.par_size[l] = g.lin_b(l, g.nh) + g.lin_out(l, g.nh);
  s.cfg = g.cfg;
  return s;
}

// warp and thread tile of a product of R rows x 128 outputs, ring depth
template <int R>
struct FlowTile {
  static constexpr int NT = R >= 64 ? 128 : 256;    // threads
  static constexpr int WR = R >= 64 ? R / 32 : 1;   // warps along the rows
  static constexpr int WC = NT / 32 / WR;           // and along the outputs
  static constexpr int TQ = R / (16 * WR);          // row quads per thread: r0 + 16 q
  static constexpr int TN = kFlowCols / (8 * WC);   // outputs per thread: c0 + 8 j
  static constexpr int LD = R + 4;                  // pitch of activations
  // two stages let two CTAs of 64 rows share an SM (their warps cover the
  // copies' latency); a 16-row tile has few warps and looks two stages ahead
  static constexpr int ST = R >= 64 ? 2 : 3;
};

// Tiles of [column][R] go to and from memory as one bulk copy per column (R
// floats, 16-byte aligned on both sides; smem pitch R + 4). A store is issued by
// the thread of its column after fence_async + barrier; the tile may be
// overwritten after the issuing threads' bulk_store_wait and a barrier.
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
template <int R>
__device__ __forceinline__ void tile_store(const float* tile, float* dst, int cols) {
  for (int c = threadIdx.x; c < cols; c += FlowTile<R>::NT)
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + (int64_t)c * R),
                 "r"((uint32_t)__cvta_generic_to_shared(tile + c * FlowTile<R>::LD)), "r"(4 * R)
                 : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// all but the `N` newest stores of this thread have read their tile
template <int N>
__device__ __forceinline__ void bulk_store_wait() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

// lanes: 4 row groups x 8 outputs
__device__ __forceinline__ int flow_lane_row() { return ((threadIdx.x & 31) >> 3) * 4; }
__device__ __forceinline__ int flow_lane_col() { return threadIdx.x & 7; }

// the stream of weight stages, in the order the products use them; a thread
// copies outputs tid / 8 + NT / 8 q at inputs 2 (tid % 8) (8-byte copies, where
// every row of W is 8-byte aligned) or tid / 16 + NT / 16 q at tid % 16 (4-byte)
template <int NT, int ST>
struct WStream {
  const FlowShape* s;
  const float* theta;
  uint32_t ring;         // shared-memory address
  int step;              // +1: layers 0 .. L-1, -1: L-1 .. 0
  int l, left, i, t, tiles, N, K, slot;
  int k;                 // this thread's input in the next stage
  const float* src;      // its first output's weight there
  bool v2;

  __device__ __forceinline__ void set() {
    const int out = s->out(l, i), tc = s->tile_cols(i);
    K = s->in(l, i);
    tiles = (out + tc - 1) / tc;
    N = min(tc, out - t * tc);
    const float* W = theta + s->layer_off(l) + s->w_off(l, i) + (int64_t)t * tc * K;
    v2 = ((uintptr_t)W & 7) == 0 && (K & 1) == 0;
    k = v2 ? 2 * (threadIdx.x & 7) : threadIdx.x & 15;
    src = W + (int64_t)(v2 ? threadIdx.x >> 3 : threadIdx.x >> 4) * K + k;
  }
  __device__ __forceinline__ void begin(const FlowShape* shape, const float* th, const float* r, bool inverse) {
    s = shape;
    theta = th;
    ring = (uint32_t)__cvta_generic_to_shared(r);
    step = inverse ? -1 : 1;
    l = inverse ? s->L - 1 : 0;
    left = s->L;
    i = t = slot = 0;
    set();
#pragma unroll
    for (int q = 0; q < ST - 1; ++q) issue();
  }
  // copy the next stage (outputs < N, inputs past K as zeros) into its ring slot
  __device__ __forceinline__ void issue() {
    if (left > 0) {
      const uint32_t dst = ring + slot * (4 * kFlowStageFloats);
      const bool in = k < K;
      const float* p = in ? src : theta;
      const int64_t row = in ? (int64_t)K : 0;
      if (v2) {
        const int n = threadIdx.x >> 3;
        const uint32_t d0 = dst + 4 * (n * kFlowPitch + 2 * (threadIdx.x & 7));
        const int bytes = in ? 8 : 0;
#pragma unroll
        for (int q = 0; q < kFlowCols * 8 / NT; ++q)
          if (n + NT / 8 * q < N)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d0 + q * (NT / 8 * 4 * kFlowPitch)),
                         "l"(p + NT / 8 * q * row), "r"(bytes));
      } else {
        const int n = threadIdx.x >> 4;
        const uint32_t d0 = dst + 4 * (n * kFlowPitch + (threadIdx.x & 15));
        const int bytes = in ? 4 : 0;
#pragma unroll
        for (int q = 0; q < kFlowCols * 16 / NT; ++q)
          if (n + NT / 16 * q < N)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d0 + q * (NT / 16 * 4 * kFlowPitch)),
                         "l"(p + NT / 16 * q * row), "r"(bytes));
      }
      slot = slot + 1 == ST ? 0 : slot + 1;
      const int k_first = k - (v2 ? 2 * (threadIdx.x & 7) : threadIdx.x & 15) + kFlowBK;   // of the stage after
      k += kFlowBK;
      src += kFlowBK;
      if (k_first >= K) {
        if (++t == tiles) {
          t = 0;
          if (++i > s->nh) {
            i = 0;
            l += step;
            --left;
          }
        }
        if (left > 0) set();
      }
    }
    asm volatile("cp.async.commit_group;");
  }
};

// One product tile: out[q][j] = the four rows r0 + 16 q .. + 3 of A . W^T for
// output c0 + 8 j, consuming ceil(K / 16) stages of the stream. A is [k][row]
// with finite values up to a multiple of 16 inputs. Every stage starts with a
// barrier.
template <int R>
__device__ __forceinline__ void flow_product(WStream<FlowTile<R>::NT, FlowTile<R>::ST>& w, const float* ring, int& slot, const float* A, int N, int K, int r0,
                                             int c0, float4 (&out)[FlowTile<R>::TQ][FlowTile<R>::TN]) {
  using T = FlowTile<R>;
  constexpr int TQ = T::TQ, TN = T::TN;
  uint64_t acc[TQ][TN][2];
#pragma unroll
  for (int q = 0; q < TQ; ++q)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[q][j][0] = acc[q][j][1] = 0ull;
  const int warp_c0 = c0 - flow_lane_col();
  const float* Ar = A + r0;
  for (int k0 = 0; k0 < K; k0 += kFlowBK) {
    asm volatile("cp.async.wait_group %0;" ::"n"(T::ST - 2) : "memory");
    __syncthreads();
    w.issue();
    if (warp_c0 < N) {
      const float* Ws = ring + slot * kFlowStageFloats + c0 * kFlowPitch;
#pragma unroll
      for (int k = 0; k < kFlowBK; k += 4) {
        float4 b[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(Ws + 8 * j * kFlowPitch + k);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          uint64_t bb[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const float v = r == 0 ? b[j].x : r == 1 ? b[j].y : r == 2 ? b[j].z : b[j].w;
            bb[j] = f2_pack(v, v);
          }
#pragma unroll
          for (int q = 0; q < TQ; ++q) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(Ar + (k + r) * T::LD + 16 * q);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
              acc[q][j][0] = f2_fma(a.x, bb[j], acc[q][j][0]);
              acc[q][j][1] = f2_fma(a.y, bb[j], acc[q][j][1]);
            }
          }
        }
      }
    }
    Ar += kFlowBK * T::LD;
    slot = slot + 1 == T::ST ? 0 : slot + 1;
  }
#pragma unroll
  for (int q = 0; q < TQ; ++q)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      f2_unpack(acc[q][j][0], out[q][j].x, out[q][j].y);
      f2_unpack(acc[q][j][1], out[q][j].z, out[q][j].w);
    }
}

// ------------------------------------------------------------------ backward products
// The stream of weight rows for C[row, n] = sum_k G[row, k] W[k, n] (a Linear's
// input gradient: k its outputs, n its inputs), layers L-1 .. 0 and Linears
// nh .. 0, in stages of 16 rows; the last Linear's rows in groups of dg
// coordinates, each padded to whole stages with zeros.
template <int NT, int ST>
struct WtStream {
  const FlowShape* s;
  const float* theta;
  uint32_t ring;
  int l, i, g0, K, N, slot, k0;   // g0: first row of the group, K: its rows
  const float* W;                 // row g0 of W
  bool v2;

  __device__ __forceinline__ void set() {
    N = s->in(l, i);
    const int out = s->out(l, i);
    K = i == s->nh ? min(s->dg * s->P, out - g0) : out;
    W = theta + s->layer_off(l) + s->w_off(l, i) + (int64_t)g0 * N;
    v2 = ((uintptr_t)W & 7) == 0 && (N & 1) == 0;
    k0 = 0;
  }
  __device__ __forceinline__ void begin(const FlowShape* shape, const float* th, const float* r) {
    s = shape;
    theta = th;
    ring = (uint32_t)__cvta_generic_to_shared(r);
    l = s->L - 1;
    i = s->nh;
    g0 = slot = 0;
    set();
#pragma unroll
    for (int q = 0; q < ST - 1; ++q) issue();
  }
  __device__ __forceinline__ void issue() {
    if (l >= 0) {
      const uint32_t dst = ring + slot * (4 * kFlowBK * kFlowCols);
      if (v2) {
        constexpr int C2 = kFlowCols / 2, RPT = NT / C2;   // 8-byte chunks per row, rows per pass
        const int r = threadIdx.x / C2, c = 2 * (threadIdx.x % C2);
        if (c < N) {
#pragma unroll
          for (int q = 0; q < kFlowBK / RPT; ++q) {
            const int rr = r + RPT * q, k = k0 + rr;
            const int bytes = k < K ? 8 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + 4 * (rr * kFlowCols + c)),
                         "l"(W + (int64_t)(k < K ? k : 0) * N + c), "r"(bytes));
          }
        }
      } else {
        constexpr int RPT = NT / kFlowCols;
        const int r = threadIdx.x / kFlowCols, c = threadIdx.x % kFlowCols;
        if (c < N) {
#pragma unroll 4
          for (int q = 0; q < kFlowBK / RPT; ++q) {
            const int rr = r + RPT * q, k = k0 + rr;
            const int bytes = k < K ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * (rr * kFlowCols + c)),
                         "l"(W + (int64_t)(k < K ? k : 0) * N + c), "r"(bytes));
          }
        }
      }
      slot = slot + 1 == ST ? 0 : slot + 1;
      k0 += kFlowBK;
      if (k0 >= K) {
        g0 += K;
        if (g0 == s->out(l, i)) {
          g0 = 0;
          if (--i < 0) {
            i = s->nh;
            --l;
          }
        }
        if (l >= 0) set();
      }
    }
    asm volatile("cp.async.commit_group;");
  }
};

// columns of a thread in the backward products: pairs or quads of adjacent
// columns, col(0) .. , groups 32 columns apart
template <int R>
struct FlowTileT {
  using T = FlowTile<R>;
  static constexpr int E = T::TN >= 4 ? 4 : T::TN;   // adjacent columns
  static constexpr int NG = T::TN / E;               // groups, 8 E columns apart
  static __device__ __forceinline__ int col0() {
    return ((threadIdx.x >> 5) % T::WC) * (8 * T::TN) + (threadIdx.x & 7) * E;
  }
};

// acc[q][c][.] += the four rows r0 + 16 q .. of G . W for this thread's TN
// columns, over K rows of W; G is [k][row] with zeros up to a multiple of 16
template <int R>
__device__ __forceinline__ void flow_product_t(WtStream<FlowTile<R>::NT, FlowTile<R>::ST>& w, const float* ring, int& slot,
                                               const float* G, int N, int K, int r0,
                                               uint64_t (&acc)[FlowTile<R>::TQ][FlowTile<R>::TN][2]) {
  using T = FlowTile<R>;
  using U = FlowTileT<R>;
  const int c0 = U::col0();
  const bool on = ((threadIdx.x >> 5) % T::WC) * (8 * T::TN) < N;
  const float* Gr = G + r0;
  for (int k0 = 0; k0 < K; k0 += kFlowBK) {
    asm volatile("cp.async.wait_group %0;" ::"n"(T::ST - 2) : "memory");
    __syncthreads();
    w.issue();
    if (on) {
      const float* Ws = ring + slot * (kFlowBK * kFlowCols) + c0;
#pragma unroll
      for (int k = 0; k < kFlowBK; ++k) {
        uint64_t b[T::TN];
#pragma unroll
        for (int g = 0; g < U::NG; ++g) {
          if constexpr (U::E == 4) {
            const float4 v = *reinterpret_cast<const float4*>(Ws + k * kFlowCols + 32 * g);
            b[4 * g] = f2_pack(v.x, v.x);
            b[4 * g + 1] = f2_pack(v.y, v.y);
            b[4 * g + 2] = f2_pack(v.z, v.z);
            b[4 * g + 3] = f2_pack(v.w, v.w);
          } else {
            const float2 v = *reinterpret_cast<const float2*>(Ws + k * kFlowCols);
            b[0] = f2_pack(v.x, v.x);
            b[1] = f2_pack(v.y, v.y);
          }
        }
#pragma unroll
        for (int q = 0; q < T::TQ; ++q) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(Gr + k * T::LD + 16 * q);
#pragma unroll
          for (int j = 0; j < T::TN; ++j) {
            acc[q][j][0] = f2_fma(a.x, b[j], acc[q][j][0]);
            acc[q][j][1] = f2_fma(a.y, b[j], acc[q][j][1]);
          }
        }
      }
    }
    Gr += kFlowBK * T::LD;
    slot = slot + 1 == T::ST ? 0 : slot + 1;
  }
}

}  // namespace fmc
