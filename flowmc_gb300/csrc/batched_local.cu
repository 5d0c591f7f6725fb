// batched_local.cu -- many independent dense-Gaussian targets of uneven
// dimension sampled in ONE persistent launch (MALA or HMC).
//
// Work items are chain tiles of one target; CTAs pull items from an atomic
// counter (a persistent scheduler, the largest dimensions first: long items
// never leave SMs idle behind short ones) and run all n_steps of their tile
// before taking the next. The gradient of log p = -0.5 dx^T P dx (dx = x -
// mean, P symmetric) is a [chains x d] x [d x d] FP32 product per evaluation,
// which is what the kernel spends its time on (FMA issue; 2 d^2 FLOPs per
// chain and evaluation against 4 d + 8 bytes per chain and step).
//
// Tile: 12 warps, each owning a 32-chain x 32-coordinate block of the product
// (8 chains x 4 coordinates per thread; lanes 4 chains x 8 coordinate groups,
// so that every 16-byte shared-memory read of a warp is conflict-free). A
// target of d coordinates takes cb = ceil(d / 32) warps side by side -- a row
// block of 32 chains -- and up to floor(12 / cb) row blocks, so that narrow
// targets fill the CTA with more chains instead of leaving threads idle.
// Positions, momenta and gradients of the trajectory are in the owner threads'
// registers (168 a thread at 12 warps, of which the HMC instance spills 164 bytes), the
// position and gradient that the chain holds in shared memory; dx is
// shared by the warps of a row block through shared memory. P, packed once per call into rows of 32 cb values, streams from L2:
// every warp copies its own 32 columns (cp.async, 8-row stages, three in
// flight, running on into the next evaluation), so no barrier is needed for
// P and the only ones in the product loop are the row block's two per
// evaluation around dx. With one ring per CTA and a CTA barrier per 16 rows
// instead, warps spent a quarter of their time at that barrier.
//
// Each product element is one FMA chain in k order, and the per-chain sums
// keep one fixed order whatever the tile shape, so the tile shape never
// changes a trajectory.
//
// Measured (48 targets of 8-256 dimensions, 146,569 chains; before: 32-chain
// tiles of 8 warps, P read from L2 into registers, all state in shared
// memory): MALA 10 steps 7.38 -> 3.03 ms, HMC 3 steps of 11
// gradients 16.4 -> 6.55 ms per call, about 30 TFLOP/s of useful FP32 (46 % of
// the FMA pipe with padding; issue slots 58 % busy, bound by the latency of the
// shared-memory reads with two or three warps per scheduler).
//
// Step semantics are those of fmc_local_steps (MALA.py:26-89, HMC.py:98-151
// with an identity mass matrix); the output of target t is written to its own
// buffers [n_chains_t, buf_len, d_t] at the clamped cursor.
#include <algorithm>
#include <string.h>
#include <vector>
#include "local_steps.cuh"

namespace fmc {

constexpr int kBWarps = 12;
constexpr int kBThreads = 32 * kBWarps;
constexpr int kBDMax = 256;
constexpr int kBRows = 32 * kBWarps;     // most chains of a tile (d <= 32)
constexpr int kBStage = 8;               // rows of P per stage
constexpr int kBStages = 4;              // stages of a warp's ring
// dx rows are padded by 4 floats (consecutive rows four banks apart); the
// largest of rows * (32 cb + 4) over the tile shapes is 384 * 36
constexpr int kBDxFloats = kBRows * 36;
constexpr int kBRing = kBStages * kBStage * 32;   // floats of one warp's ring
constexpr int kBPartFloats = kBWarps * 32 * 8;

struct BatchTarget {
  const float* precision;   // [d, d]
  float* packed;            // [round_up(d, 8), round_up(d, 32)] (k_pack_precision)
  const float* mean;        // [d] or NULL
  float const_term;
  int d;
  int n_chains;
  int tile_rows;            // chains per work item (a multiple of 32)
  int chain_offset;         // first row of this target in x0 / x_last / lp_last ([sum C, 256])
  float* out_pos;           // [n_chains, buf_len, d]
  float* out_logp;          // [n_chains, buf_len]
  float* out_acc;
  float step;
  const float* noise;       // [n_chains, n_steps, d] explicit normals or NULL
  const float* unif;        // [n_chains, n_steps] explicit uniforms or NULL
};

struct BatchArgs {
  const BatchTarget* targets;
  const int32_t* item_target;   // [n_items]
  const int32_t* item_chain0;   // [n_items]
  int n_items;
  int* next_item;               // scheduler counter (zeroed before the launch)
  int n_leapfrog, S, thin;
  int64_t buf_len, start;
  Rng rng;
  const float* x0;              // [sum C, 256] (row stride 256)
  float* x_last;                // [sum C, 256]
  float* lp_last;               // [sum C]
};

constexpr size_t kBSmemBytes =
    sizeof(float) * (2 * 8 * 4 * (size_t)kBThreads + kBDxFloats + kBWarps * kBRing + kBPartFloats + 7 * (size_t)kBRows);
static_assert(kBSmemBytes <= 227 * 1024, "shared memory");

// The precision matrices in the layout the product streams: [8 ns][32 cb]
// with zeros outside [d, d], so that every stage of 8 rows is one contiguous
// 16-byte aligned block whatever d is.
__global__ void k_pack_precision(const BatchTarget* __restrict__ targets) {
  const BatchTarget T = targets[blockIdx.x];
  const int w = (T.d + 31) & ~31, kp = (T.d + kBStage - 1) & ~(kBStage - 1);
  for (int k = blockIdx.y; k < kp; k += gridDim.y)
    for (int j = threadIdx.x; j < w; j += blockDim.x)
      T.packed[k * w + j] = (k < T.d && j < T.d) ? __ldg(T.precision + (int64_t)k * T.d + j) : 0.f;
}

// This thread's place in the tile and its row block's shared memory.
struct BatchBlock {
  int cb;         // warps (32-coordinate blocks) of the row block
  int tb;         // thread index within the row block's 32 cb threads
  int bar;        // the row block's named barrier
  int r0;         // this thread's chains: r0 + 4 c of the row block's 32
  int j0;         // its coordinates: j0 .. j0 + 3
  int ldx;
  float* DX;      // [32][ldx]
  float* part;    // [32][8 cb] per-thread partials of dx . P dx
  float* ring;    // this warp's P stages
  const float* src;   // its 16 bytes of the packed P's row (lane / 8), column block first
  int ns, next, buf;  // stages of P, next stage to copy, ring slot to read
  float4 mean;
  __device__ __forceinline__ void sync() const {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * cb) : "memory");
  }
  // copy the next stage (8 rows x this warp's 32 columns) into `slot`
  __device__ __forceinline__ void issue(int slot) {
    const int lane = threadIdx.x & 31, w = 32 * cb;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + slot * (kBStage * 32)) + 16 * lane;
    const float* p = src + next * kBStage * w;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512), "l"(p + 4 * w));
    asm volatile("cp.async.commit_group;");
    next = next + 1 == ns ? 0 : next + 1;
  }
};

// g[c][.] = -(dx P) of this thread's 8 chains x 4 coordinates at positions y;
// with lp != NULL also lp[row] = -0.5 dx . P dx + const for the row block's
// chains. The caller's row block has passed a barrier since its last use of
// DX; on return DX may still be read by other warps unless lp is given.
__device__ __forceinline__ void dense_eval(const BatchTarget& T, BatchBlock& B, const float (&y)[8][4],
                                           float (&g)[8][4], float* lp) {
  const int d = T.d, ldx = B.ldx, j0 = B.j0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    // dx = x - mean, zero on the padding coordinates
    float4 v;
    v.x = j0 + 0 < d ? y[c][0] - B.mean.x : 0.f;
    v.y = j0 + 1 < d ? y[c][1] - B.mean.y : 0.f;
    v.z = j0 + 2 < d ? y[c][2] - B.mean.z : 0.f;
    v.w = j0 + 3 < d ? y[c][3] - B.mean.w : 0.f;
    *reinterpret_cast<float4*>(B.DX + (B.r0 + 4 * c) * ldx + j0) = v;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int u = 0; u < 4; ++u) g[c][u] = 0.f;
  B.sync();
  const float* Xs = B.DX + B.r0 * ldx;
#pragma unroll 1
  for (int s = 0; s < B.ns; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kBStages - 2) : "memory");
    __syncwarp();
    // the slot read in the previous iteration, which every lane has left
    B.issue((B.buf + kBStages - 1) % kBStages);
    const float* Ps = B.ring + B.buf * (kBStage * 32) + (threadIdx.x & 7) * 4;
    // rows of the packed P past d are zero; dx has zeros there too
#pragma unroll
    for (int k = 0; k < kBStage; k += 4) {
      float4 p[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) p[r] = *reinterpret_cast<const float4*>(Ps + (k + r) * 32);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 x = *reinterpret_cast<const float4*>(Xs + 4 * c * ldx + k);
        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          g[c][0] = fmaf(xv[r], p[r].x, g[c][0]);
          g[c][1] = fmaf(xv[r], p[r].y, g[c][1]);
          g[c][2] = fmaf(xv[r], p[r].z, g[c][2]);
          g[c][3] = fmaf(xv[r], p[r].w, g[c][3]);
        }
      }
    }
    Xs += kBStage;
    B.buf = (B.buf + 1) % kBStages;
  }
  if (lp != nullptr) {
    const int nj = 8 * B.cb;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 v = *reinterpret_cast<const float4*>(B.DX + (B.r0 + 4 * c) * ldx + j0);
      const float xv[4] = {v.x, v.y, v.z, v.w};
      float q = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + u < d) q = fmaf(xv[u], g[c][u], q);
      B.part[(B.r0 + 4 * c) * nj + (j0 >> 2)] = q;
    }
    B.sync();
    // per chain: the partials of the 64 coordinate groups (absent ones zero)
    // as two balanced trees of 32, eight lanes per chain
    const int sub = B.tb & 7;
    for (int r = B.tb >> 3; r < 32; r += 4 * B.cb) {
      const float* pr = B.part + r * nj;
      float h[2];
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = 32 * b + sub + 8 * q;
          v[q] = i < nj ? pr[i] : 0.f;
        }
        float t = (v[0] + v[2]) + (v[1] + v[3]);
        t += __shfl_xor_sync(0xffffffffu, t, 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        h[b] = t;
      }
      if (sub == 0) lp[r] = -0.5f * (h[0] + h[1]) + T.const_term;
    }
    B.sync();
  }
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int u = 0; u < 4; ++u) g[c][u] = -g[c][u];
}

// out[r] = sum over j < d of DX[r][j]^2 for the row block, where DX holds v:
// eight lanes per chain (lane sub takes j = sub, sub + 8, ...), then a
// three-level butterfly. Barriers before the write, after it and at the end.
__device__ __forceinline__ void row_sumsq(const BatchTarget& T, const BatchBlock& B, const float (&v)[8][4],
                                          float* out) {
  B.sync();
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(B.DX + (B.r0 + 4 * c) * B.ldx + B.j0) = make_float4(v[c][0], v[c][1], v[c][2], v[c][3]);
  B.sync();
  const int sub = B.tb & 7;
  for (int r = B.tb >> 3; r < 32; r += 4 * B.cb) {
    const float* e = B.DX + r * B.ldx;
    float t = 0.f;
    for (int j = sub; j < T.d; j += 8) t = fmaf(e[j], e[j], t);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    if (sub == 0) out[r] = t;
  }
  B.sync();
}

// normals of chain c of T at step s for coordinates j0 .. j0 + 3 (j0 a
// multiple of 4): explicit, or component j & 1 of the Box-Muller pair of the
// Philox block keyed by j >> 1
__device__ __forceinline__ void draw_normals4(const BatchArgs& a, const Rng& rng, const BatchTarget& T, int c, int s,
                                              int j0, float (&xi)[4]) {
  if (T.noise) {
    const float* row = T.noise + ((int64_t)c * a.S + s) * T.d + j0;
#pragma unroll
    for (int u = 0; u < 4; ++u) xi[u] = (c < T.n_chains && j0 + u < T.d) ? __ldg(row + u) : 0.f;
    return;
  }
#pragma unroll
  for (int u = 0; u < 4; u += 2) {
    const u32x4 r = rng.draw((uint64_t)(T.chain_offset + c), (uint64_t)s, (uint32_t)((j0 + u) >> 1),
                             RNG_TAG_LOCAL_NORMAL);
    box_muller(r.x, r.y, xi[u], xi[u + 1]);
  }
}

// all steps of one work item for this thread's row block
template <int KIND>
__device__ __forceinline__ void run_tile(const BatchArgs& a, const Rng& rng, const BatchTarget& T, BatchBlock& B, int c0,
                                         int nc, float4* sx, float4* sg, float* chain) {
  // per-chain values of the row block, kBRows apart
  float *lpx = chain, *lpy = chain + kBRows, *sA = chain + 2 * kBRows, *sB = chain + 3 * kBRows;
  float* logu = chain + 4 * kBRows;
  int* acc_s = reinterpret_cast<int*>(chain + 5 * kBRows);
  const int d = T.d, j0 = B.j0, s_rec = (a.S - 1) / a.thin * a.thin;   // s_rec: the last recorded step
  const bool vec_out = (d & 3) == 0 && ((uintptr_t)T.out_pos & 15) == 0;
  const float dt = T.step, dt2 = dt * dt;
  float y[8][4], g[8][4];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int r = B.r0 + 4 * c;
    const float* xr = a.x0 + (int64_t)(T.chain_offset + c0 + r) * kBDMax + j0;
#pragma unroll
    for (int u = 0; u < 4; ++u) y[c][u] = (r < nc && j0 + u < d) ? xr[u] : 0.f;
    sx[c * kBThreads] = make_float4(y[c][0], y[c][1], y[c][2], y[c][3]);
  }
  dense_eval(T, B, y, g, lpx);
#pragma unroll
  for (int c = 0; c < 8; ++c) sg[c * kBThreads] = make_float4(g[c][0], g[c][1], g[c][2], g[c][3]);

  for (int s = 0; s < a.S; ++s) {
    // log-uniforms of the step, one chain per thread
    if (B.tb < nc && B.tb < 32) {
      const int64_t row = c0 + B.tb;
      float u;
      if (T.unif) u = __ldg(T.unif + row * a.S + s);
      else u = u32_to_unit(rng.draw((uint64_t)(T.chain_offset + row), (uint64_t)s, 0u, RNG_TAG_LOCAL_UNIFORM).x);
      logu[B.tb] = logf(u);
    }
    // ---- proposal (MALA) or leapfrog trajectory (HMC): y, g, lpy
    if constexpr (KIND == FMC_KERNEL_MALA) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float xi[4];
        draw_normals4(a, rng, T, c0 + B.r0 + 4 * c, s, j0, xi);
        const float4 x = sx[c * kBThreads], gx = sg[c * kBThreads];
        y[c][0] = fmaf(dt, xi[0], x.x + dt2 * gx.x / 2.0f);
        y[c][1] = fmaf(dt, xi[1], x.y + dt2 * gx.y / 2.0f);
        y[c][2] = fmaf(dt, xi[2], x.z + dt2 * gx.z / 2.0f);
        y[c][3] = fmaf(dt, xi[3], x.w + dt2 * gx.w / 2.0f);
      }
      dense_eval(T, B, y, g, lpy);
      // |prop - mean0|^2 and |x - mean1|^2 per chain
      float e[8][4];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 x = sx[c * kBThreads], gx = sg[c * kBThreads];
        e[c][0] = y[c][0] - (x.x + dt2 * gx.x / 2.0f);
        e[c][1] = y[c][1] - (x.y + dt2 * gx.y / 2.0f);
        e[c][2] = y[c][2] - (x.z + dt2 * gx.z / 2.0f);
        e[c][3] = y[c][3] - (x.w + dt2 * gx.w / 2.0f);
      }
      row_sumsq(T, B, e, sA);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 x = sx[c * kBThreads];
        e[c][0] = x.x - (y[c][0] + dt2 * g[c][0] / 2.0f);
        e[c][1] = x.y - (y[c][1] + dt2 * g[c][1] / 2.0f);
        e[c][2] = x.z - (y[c][2] + dt2 * g[c][2] / 2.0f);
        e[c][3] = x.w - (y[c][3] + dt2 * g[c][3] / 2.0f);
      }
      row_sumsq(T, B, e, sB);
    } else {
      float p[8][4];
#pragma unroll
      for (int c = 0; c < 8; ++c) draw_normals4(a, rng, T, c0 + B.r0 + 4 * c, s, j0, p[c]);
      row_sumsq(T, B, p, sA);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 x = sx[c * kBThreads], gx = sg[c * kBThreads];
        y[c][0] = x.x; y[c][1] = x.y; y[c][2] = x.z; y[c][3] = x.w;
        // row 0: half kick with the gradient at x
        p[c][0] = fmaf(dt * 0.5f, gx.x, p[c][0]);
        p[c][1] = fmaf(dt * 0.5f, gx.y, p[c][1]);
        p[c][2] = fmaf(dt * 0.5f, gx.z, p[c][2]);
        p[c][3] = fmaf(dt * 0.5f, gx.w, p[c][3]);
      }
      for (int r = 1; r <= a.n_leapfrog + 1; ++r) {
        const bool end = r == a.n_leapfrog + 1;
        const float ek = end ? dt * 0.5f : dt;
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
          for (int u = 0; u < 4; ++u) y[c][u] = fmaf(dt, p[c][u], y[c][u]);
        if (r > 1) B.sync();   // every warp has left the previous product's dx
        // only the gradient is used before the end point
        dense_eval(T, B, y, g, end ? lpy : nullptr);
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
          for (int u = 0; u < 4; ++u) p[c][u] = fmaf(ek, g[c][u], p[c][u]);
      }
      row_sumsq(T, B, p, sB);
    }
    // ---- accept per chain (float-float log-ratio), then commit
    const bool rec = s % a.thin == 0;
    const int64_t orow = a.start + s / a.thin;
    if (B.tb < nc && B.tb < 32) {
      const int c = B.tb;
      ff ratio;
      if constexpr (KIND == FMC_KERNEL_MALA) {
        const ff q = two_sum(sA[c], -sB[c]);
        ratio = ff_add(two_sum(lpy[c], -lpx[c]), ff_mul_f(q, 0.5f / (dt * dt)));
      } else {
        ratio = ff_add(two_sum(-lpx[c], 0.5f * sA[c]), ff_neg(two_sum(-lpy[c], 0.5f * sB[c])));
      }
      const bool acc = f_lt_ff(logu[c], ratio);
      acc_s[c] = acc ? 1 : 0;
      const float lp = acc ? lpy[c] : lpx[c];
      lpx[c] = lp;
      if (rec) {
        __stcs(T.out_logp + (int64_t)(c0 + c) * a.buf_len + orow, lp);
        __stcs(T.out_acc + (int64_t)(c0 + c) * a.buf_len + orow, acc ? 1.f : 0.f);
        if (s == s_rec) a.lp_last[T.chain_offset + c0 + c] = lp;
      }
    }
    B.sync();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int r = B.r0 + 4 * c;
      if (r >= nc) continue;
      if (acc_s[r]) {
        sx[c * kBThreads] = make_float4(y[c][0], y[c][1], y[c][2], y[c][3]);
        sg[c * kBThreads] = make_float4(g[c][0], g[c][1], g[c][2], g[c][3]);
      }
      if (rec && j0 < d) {
        const float4 x = sx[c * kBThreads];
        const float xv[4] = {x.x, x.y, x.z, x.w};
        float* o = T.out_pos + ((int64_t)(c0 + r) * a.buf_len + orow) * d + j0;
        if (vec_out) {
          __stcs(reinterpret_cast<float4*>(o), x);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (j0 + u < d) __stcs(o + u, xv[u]);
        }
        if (s == s_rec) {
          float* xl = a.x_last + (int64_t)(T.chain_offset + c0 + r) * kBDMax + j0;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (j0 + u < d) xl[u] = xv[u];
        }
      }
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(kBThreads, 1) k_batched_dense(const BatchArgs a) {
  extern __shared__ __align__(16) float smraw[];
  const Rng rng = a.rng.at_epoch();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  float4* sx = reinterpret_cast<float4*>(smraw) + tid;   // [8][kBThreads] positions, owner thread's layout
  float4* sg = sx + 8 * kBThreads;                       // gradients at those positions
  float* DX = smraw + 2 * 8 * 4 * kBThreads;
  float* ring = DX + kBDxFloats;
  float* part = ring + kBWarps * kBRing;
  float* chain = part + kBPartFloats;
  __shared__ int item_s;

  for (;;) {
    if (tid == 0) item_s = atomicAdd(a.next_item, 1);
    __syncthreads();
    const int item = item_s;
    if (item >= a.n_items) break;
    const BatchTarget T = a.targets[a.item_target[item]];
    const int c0 = a.item_chain0[item];
    const int nc = min(T.tile_rows, T.n_chains - c0);
    BatchBlock B;
    B.cb = (T.d + 31) >> 5;
    const int rb = wid / B.cb, wb = wid - rb * B.cb;   // row block, coordinate block
    if (32 * rb < nc) {
      B.tb = wb * 32 + lane;
      B.bar = 1 + rb;
      B.r0 = lane >> 3;
      B.j0 = wb * 32 + (lane & 7) * 4;
      B.ldx = 32 * B.cb + 4;
      B.DX = DX + 32 * rb * B.ldx;
      B.part = part + 32 * rb * 8 * B.cb;
      B.ring = ring + wid * kBRing;
      B.src = T.packed + (lane >> 3) * 32 * B.cb + B.j0;
      B.ns = (T.d + kBStage - 1) / kBStage;
      B.next = 0;
      B.buf = 0;
      B.mean = make_float4(0.f, 0.f, 0.f, 0.f);
      if (T.mean != nullptr) {
        if (B.j0 + 0 < T.d) B.mean.x = __ldg(T.mean + B.j0);
        if (B.j0 + 1 < T.d) B.mean.y = __ldg(T.mean + B.j0 + 1);
        if (B.j0 + 2 < T.d) B.mean.z = __ldg(T.mean + B.j0 + 2);
        if (B.j0 + 3 < T.d) B.mean.w = __ldg(T.mean + B.j0 + 3);
      }
#pragma unroll
      for (int q = 0; q < kBStages - 1; ++q) B.issue(q);
      run_tile<KIND>(a, rng, T, B, c0 + 32 * rb, nc - 32 * rb, sx, sg, chain + 32 * rb);
      asm volatile("cp.async.wait_group 0;" ::: "memory");   // the stages copied ahead
    }
    __syncthreads();   // item_s and the shared buffers are free
  }
}

// Chains per work item for each target: up to floor(12 / cb) blocks of 32
// chains (at most `cap`), where cb = ceil(d / 32) warps stand side by side.
static int batch_tile_rows(int d, int n_chains, int cap) {
  const int cb = (d + 31) / 32;
  int rb = kBWarps / cb;
  if (rb > cap) rb = cap;
  const int need = (n_chains + 31) / 32;
  if (rb > need) rb = need;
  return 32 * rb;
}

}  // namespace fmc

using namespace fmc;

// Positions of up to kPackTargets targets into the padded layout: target
// blockIdx.y, one warp per row. One launch where a copy per target took 48 for
// 48 targets (160 us of launches for 50 MB); the table travels as the
// kernel's parameters.
constexpr int kPackTargets = 64;
struct PackRows {
  const float* x[kPackTargets];
  int64_t ld[kPackTargets];
  int64_t row0[kPackTargets];   // first row in the padded layout
  int32_t n[kPackTargets], d[kPackTargets];
};
__global__ void __launch_bounds__(256) k_pack_rows(const __grid_constant__ PackRows a, float* __restrict__ out) {
  const int t = blockIdx.y, lane = threadIdx.x & 31, d = a.d[t], n = a.n[t];
  const float* x = a.x[t];
  const int64_t ld = a.ld[t];
  float* o = out + a.row0[t] * kBDMax;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < n; r += gridDim.x * 8)
    for (int j = lane; j < d; j += 32) o[(int64_t)r * kBDMax + j] = x[r * ld + j];
}

extern "C" int fmc_batched_pack_rows(const float* const* x, const int64_t* row_stride, const int32_t* n_dim,
                                     const int32_t* n_chains, int32_t n_targets, float* packed, void* stream) {
  FMC_CHECK_ARG(x && row_stride && n_dim && n_chains && packed && n_targets >= 1, "bad arguments");
  int64_t row = 0;
  for (int t0 = 0; t0 < n_targets; t0 += kPackTargets) {
    PackRows a{};
    const int nt = n_targets - t0 < kPackTargets ? n_targets - t0 : kPackTargets;
    int most = 1;
    for (int i = 0; i < nt; ++i) {
      const int t = t0 + i;
      FMC_CHECK_ARG(x[t] && n_chains[t] >= 1 && n_dim[t] >= 1 && n_dim[t] <= kBDMax, "target %d: bad rows", t);
      a.x[i] = x[t];
      a.ld[i] = row_stride[t];
      a.row0[i] = row;
      a.n[i] = n_chains[t];
      a.d[i] = n_dim[t];
      row += n_chains[t];
      if (n_chains[t] > most) most = n_chains[t];
    }
    const int bx = (most + 15) / 16 < 256 ? (most + 15) / 16 : 256;   // two rows a warp, or more
    k_pack_rows<<<dim3((unsigned)bx, (unsigned)nt), 256, 0, (cudaStream_t)stream>>>(a, packed);
    FMC_LAUNCH_CHECK();
  }
  return FMC_OK;
}

// workspace without the packed precision matrices: counter, targets, work items
static size_t batched_table_bytes(int32_t n_targets, int64_t total_chains) {
  const int64_t items = total_chains / 32 + n_targets;   // at least 32 chains per work item
  return (size_t)(256 + n_targets * sizeof(BatchTarget) + 256 + items * 8 + 256);
}

// floats of a packed precision matrix (k_pack_precision)
static size_t packed_floats(int d) { return (size_t)((d + kBStage - 1) & ~(kBStage - 1)) * ((d + 31) & ~31); }

extern "C" int fmc_batched_workspace_size(int32_t n_targets, int64_t total_chains, size_t* bytes) {
  FMC_CHECK_ARG(bytes && n_targets >= 1 && total_chains >= 1, "bad arguments");
  *bytes = batched_table_bytes(n_targets, total_chains) + (size_t)n_targets * packed_floats(kBDMax) * sizeof(float);
  return FMC_OK;
}

extern "C" int fmc_batched_dense_workspace_size(const int32_t* n_dim, const int32_t* n_chains, int32_t n_targets,
                                                size_t* bytes) {
  FMC_CHECK_ARG(bytes && n_dim && n_chains && n_targets >= 1, "bad arguments");
  int64_t total = 0;
  size_t floats = 0;
  for (int t = 0; t < n_targets; ++t) {
    FMC_CHECK_ARG(n_dim[t] >= 1 && n_dim[t] <= kBDMax, "target %d: n_dim %d outside [1, %d]", t, n_dim[t], kBDMax);
    FMC_CHECK_ARG(n_chains[t] >= 1, "target %d: no chains", t);
    total += n_chains[t];
    floats += packed_floats(n_dim[t]);
  }
  *bytes = batched_table_bytes(n_targets, total) + floats * sizeof(float);
  return FMC_OK;
}

extern "C" int fmc_batched_dense_local_steps(const FmcTarget* targets, int32_t n_targets, const int32_t* n_chains,
                                             const FmcLocalParams* params, const float* step_sizes,
                                             const float* x0, int32_t n_steps, int32_t thinning, uint64_t seed,
                                             uint64_t counter, const float* const* noise, const float* const* unif,
                                             float* const* out_pos, float* const* out_logp,
                                             float* const* out_acc, int64_t buf_len, int64_t cursor, float* x_last,
                                             float* lp_last, void* ws, size_t ws_bytes, void* stream) {
  FMC_CHECK_ARG(targets && n_chains && params && step_sizes && out_pos && out_logp && out_acc, "NULL host array");
  FMC_CHECK_ARG(n_targets >= 1, "n_targets < 1");
  FMC_CHECK_ARG(params->kind == FMC_KERNEL_MALA || params->kind == FMC_KERNEL_HMC,
                "batched dense targets run MALA or HMC");
  FMC_CHECK_ARG(params->kind != FMC_KERNEL_HMC || params->n_leapfrog >= 0, "n_leapfrog < 0");
  FMC_CHECK_ARG(n_steps >= 1 && thinning >= 1 && cursor >= 0, "bad step arguments");
  const int64_t n_rec = ((int64_t)n_steps + thinning - 1) / thinning;
  FMC_CHECK_ARG(n_rec <= buf_len, "update of %lld rows does not fit a buffer of %lld rows", (long long)n_rec,
                (long long)buf_len);
  FMC_CHECK_ARG(x0 && x_last && lp_last, "NULL device array");
  std::vector<BatchTarget> bt(n_targets);
  int64_t off = 0;
  size_t floats = 0;   // of the packed precision matrices
  for (int t = 0; t < n_targets; ++t) {
    const FmcTarget& g = targets[t];
    FMC_CHECK_ARG(g.kind == FMC_TARGET_DENSE_GAUSSIAN, "target %d is not a dense Gaussian", t);
    FMC_CHECK_ARG(g.n_dim >= 1 && g.n_dim <= kBDMax, "target %d: n_dim %d outside [1, %d]", t, g.n_dim, kBDMax);
    FMC_CHECK_ARG(g.precision != nullptr, "target %d: no precision matrix", t);
    FMC_CHECK_ARG(n_chains[t] >= 1, "target %d: no chains", t);
    FMC_CHECK_ARG(out_pos[t] && out_logp[t] && out_acc[t], "target %d: NULL output buffer", t);
    bt[t] = BatchTarget{g.precision, nullptr, g.mean, g.scalars[0], g.n_dim, n_chains[t], 0, (int)off,
                        out_pos[t], out_logp[t], out_acc[t], step_sizes[t],
                        noise ? noise[t] : nullptr, unif ? unif[t] : nullptr};
    off += n_chains[t];
    floats += packed_floats(g.n_dim);
  }
  const size_t need = batched_table_bytes(n_targets, off) + floats * sizeof(float);
  FMC_CHECK_ARG(ws && ws_bytes >= need, "workspace of %zu bytes < %zu needed", ws_bytes, need);
  cudaStream_t st = (cudaStream_t)stream;
  // Tile height: the most chain blocks per item that still spread over the
  // SMs. A tile of w warps takes about ceil(w / 4) * 45 d + 2000 cycles per
  // evaluation (w / 4 warps per scheduler, 32 FMAs per k at about 0.7 of the
  // issue rate, and the evaluation's barriers); the launch takes the larger
  // of the mean load per SM and the longest item.
  const int sms = sm_count();
  int best_cap = kBWarps;
  double best = 0.0;
  for (int cap : {12, 6, 4, 3, 2, 1}) {
    double total = 0.0, longest = 0.0;
    for (int t = 0; t < n_targets; ++t) {
      const int rows = batch_tile_rows(bt[t].d, n_chains[t], cap);
      const int w = rows / 32 * ((bt[t].d + 31) / 32);
      const double cost = (w + 3) / 4 * 45.0 * bt[t].d + 2000.0;
      total += cost * ((n_chains[t] + rows - 1) / rows);
      if (cost > longest) longest = cost;
    }
    const double est = total / sms > longest ? total / sms : longest;
    if (cap == kBWarps || est < 0.98 * best) {
      best = est;
      best_cap = cap;
    }
  }
  // items, the largest dimensions first
  std::vector<int> order(n_targets);
  for (int t = 0; t < n_targets; ++t) order[t] = t;
  std::stable_sort(order.begin(), order.end(), [&](int p, int q) { return bt[p].d > bt[q].d; });
  std::vector<int32_t> it, ic;
  for (int t : order) {
    bt[t].tile_rows = batch_tile_rows(bt[t].d, n_chains[t], best_cap);
    for (int c = 0; c < n_chains[t]; c += bt[t].tile_rows) {
      it.push_back(t);
      ic.push_back(c);
    }
  }
  // scheduler counter, targets and items go up as one copy; copies from
  // pageable memory are staged before cudaMemcpyAsync returns, so the host
  // vector may go out of scope
  const size_t tb = (n_targets * sizeof(BatchTarget) + 255) / 256 * 256;
  float* packed = (float*)(((uintptr_t)ws + 256 + tb + it.size() * 8 + 15) & ~(uintptr_t)15);
  for (int t = 0; t < n_targets; ++t) {
    bt[t].packed = packed;   // whole 32-float rows: 16-byte aligned
    packed += packed_floats(bt[t].d);
  }
  std::vector<char> up(256 + tb + it.size() * 8, 0);
  memcpy(up.data() + 256, bt.data(), n_targets * sizeof(BatchTarget));
  memcpy(up.data() + 256 + tb, it.data(), it.size() * 4);
  memcpy(up.data() + 256 + tb + it.size() * 4, ic.data(), ic.size() * 4);
  char* p = (char*)ws;
  FMC_CUDA_TRY(cudaMemcpyAsync(p, up.data(), up.size(), cudaMemcpyHostToDevice, st));
  BatchArgs a{};
  a.targets = (const BatchTarget*)(p + 256);
  a.item_target = (const int32_t*)(p + 256 + tb);
  a.item_chain0 = a.item_target + it.size();
  a.n_items = (int)it.size();
  a.next_item = (int*)p;
  a.n_leapfrog = params->n_leapfrog;
  a.S = n_steps;
  a.thin = thinning;
  a.buf_len = buf_len;
  a.start = cursor < buf_len - n_rec ? cursor : buf_len - n_rec;
  a.rng = Rng{(uint32_t)seed, (uint32_t)(seed >> 32), counter, rng_epoch()};
  a.x0 = x0;
  a.x_last = x_last;
  a.lp_last = lp_last;
  k_pack_precision<<<dim3((unsigned)n_targets, 16), 256, 0, st>>>(a.targets);
  FMC_LAUNCH_CHECK();
  auto kern = params->kind == FMC_KERNEL_MALA ? k_batched_dense<FMC_KERNEL_MALA> : k_batched_dense<FMC_KERNEL_HMC>;
  FMC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBSmemBytes));
  const int grid = a.n_items < sms ? a.n_items : sms;
  kern<<<grid, kBThreads, kBSmemBytes, st>>>(a);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}
