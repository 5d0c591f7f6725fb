// nf_global.cu -- K5: the NFProposal global step (resource/kernel/NF_proposal.py:27-172)
// for all chains at once.
//
//   1. flow sample of n_chains * n_steps proposals (rqSpline.py:490-496;
//      base normals from Philox or explicit)
//   2. flow log_prob of the proposals and of the current positions in one
//      pass (NF_proposal.py:44, 165-166: the proposals' flow density is
//      recomputed by the forward pass, not taken from the inverse)
//   3. k_nf_accept or k_nf_walk: the target log-density of each proposal, each chain's
//      sequential independent-MH scan (NF_proposal.py:91-126) and the thinned
//      buffer writes, fused in one kernel.
#include <algorithm>
#include "flow.cuh"
#include "targets.cuh"

namespace fmc {

int flow_apply_logprob(const FmcFlow* f, const float* x, int64_t n, float* logp, void* ws, size_t ws_bytes,
                       cudaStream_t st);
int flow_sample_rows(const FmcFlow* f, uint64_t seed, uint64_t counter, const float* z, int64_t n, float* x, void* ws,
                     size_t ws_bytes, cudaStream_t st);
size_t flow_infer_ws_bytes(const FmcFlow* f, int64_t n);

struct NfArgs {
  FmcTarget tgt;
  const float* x0;      // [C, d]
  const float* props;   // [C*S, d]
  const float* lnf;     // [C*S + C]: proposals then current positions
  int32_t C, d, S, thin;
  Rng rng;
  const float* unif;
  float *out_pos, *out_logp, *out_acc;
  int64_t buf_len, start;
  float *x_last, *lp_last;
  int32_t chains_per_block;
  int32_t round_steps;   // steps of a round: min(S, kNfSteps)
  int32_t tab_smem;   // diag Gaussian / mixture: tables staged in shared memory
  int32_t scan_off;   // floats of dynamic shared memory before the scan's arrays
  int32_t vec;        // rows are whole 16-byte chunks everywhere
};

// The accept scan. Only the scan itself is sequential, and it needs three
// numbers per proposal, so a block takes CB chains and, a round of up to kNfSteps
// steps at a time: (1) its lane groups evaluate the proposals' target log-densities in
// parallel, (2) one thread per chain runs the accepts over shared memory and
// notes which proposal each step holds, (3) the groups copy those rows to the
// buffers. A group walking its chain's steps one after the other (k_nf_walk) waits
// for a proposal's row and a full evaluation at every step: 4096 chains x 50
// steps of the 64-D mixture 160 -> 78 us, 20 chains x 30 steps of the 5-D dual moon
// 30 -> 8 us (GB300). Bound by HBM for many chains, by one evaluation and the scan's
// dependent chain for few.
constexpr int kNfSteps = 64;

template <int TGT, int G, int V>
__global__ void __launch_bounds__(256) k_nf_accept(const NfArgs a) {
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, gl = tid % G, gib = tid / G, gpb = blockDim.x / G;
  const int d = a.d, CB = a.chains_per_block;
  float* stage = nullptr;
  const TargetConst<TGT> tc(a.tgt);
  if constexpr (TGT == FMC_TARGET_DENSE_GAUSSIAN) {
    stage = smem + gib * d;
  } else if constexpr (TGT == FMC_TARGET_DIAG_GAUSSIAN || TGT == FMC_TARGET_GAUSS_MIXTURE) {
    if (a.tab_smem) {
      stage_target_table<G, V>(a.tgt, smem);
      stage = smem;
    }
  }
  const int pitch = a.round_steps | 1, n = CB * pitch;   // odd: the scan's threads on different banks
  float* lp_s = smem + a.scan_off;          // [CB][pitch] per proposal
  float* lnf_s = lp_s + n;
  float* logu_s = lnf_s + n;
  int* held_s = reinterpret_cast<int*>(logu_s + n);   // step whose proposal is held (-1: the start), * 2 + accepted
  float* cur_lp = reinterpret_cast<float*>(held_s + n);   // [CB] state of the scan
  float* cur_lnf = cur_lp + CB;
  float* rec_lp = cur_lnf + CB;             // at the last recorded step
  int* cur = reinterpret_cast<int*>(rec_lp + CB);
  int* rec = cur + CB;
  const Rng rng = a.rng.at_epoch();

  for (int64_t c0 = (int64_t)blockIdx.x * CB; c0 < a.C; c0 += (int64_t)gridDim.x * CB) {
    const int nb = (int)(a.C - c0 < CB ? a.C - c0 : CB);
    __syncthreads();
    // log-density at the current positions (take_steps.py:201-203); the loops
    // below run whole warps (the evaluations shuffle within a group)
    for (int i0 = 0; i0 < nb; i0 += gpb) {
      const bool act = i0 + gib < nb;
      const int i = act ? i0 + gib : 0;
      float x[V], g[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int j = gl * V + v;
        x[v] = (j < d) ? __ldg(a.x0 + (c0 + i) * d + j) : 0.f;
      }
      const float lp = target_eval<TGT, G, V, false>(a.tgt, tc, x, g, gl, stage);
      if (act && gl == 0) {
        cur_lp[i] = lp;
        rec_lp[i] = lp;
        cur_lnf[i] = __ldg(a.lnf + (int64_t)a.C * a.S + c0 + i);
        cur[i] = -1;
        rec[i] = -1;
      }
    }
    for (int s0 = 0; s0 < a.S; s0 += a.round_steps) {
      const int ns = min(a.round_steps, a.S - s0);
      const int items = nb * ns;
      for (int i0 = 0; i0 < items; i0 += gpb) {
        const bool act = i0 + gib < items;
        const int i = act ? i0 + gib : 0;
        const int ci = i / ns, si = i - ci * ns;
        const int64_t c = c0 + ci, row = c * a.S + s0 + si;
        float p[V], g[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int j = gl * V + v;
          p[v] = (j < d) ? __ldg(a.props + row * d + j) : 0.f;
        }
        const float lpp = target_eval<TGT, G, V, false>(a.tgt, tc, p, g, gl, stage);
        if (act && gl == 0) {
          const int q = ci * pitch + si;
          lp_s[q] = lpp;
          lnf_s[q] = __ldg(a.lnf + row);
          logu_s[q] = logf(a.unif ? __ldg(a.unif + row)
                                  : u32_to_unit(rng.draw(c, s0 + si, 0u, RNG_TAG_NF_UNIFORM).x));
        }
      }
      __syncthreads();
      if (tid < nb) {
        float lp = cur_lp[tid], lnf = cur_lnf[tid];
        int held = cur[tid];
        for (int si = 0; si < ns; ++si) {
          const int q = tid * pitch + si;
          const float lpp = lp_s[q], lnfp = lnf_s[q];
          // ratio = (lp_p - lp_c) - (lnf_p - lnf_c)   (NF_proposal.py:102-104)
          const ff ratio = ff_add(two_sum(lpp, -lp), ff_neg(two_sum(lnfp, -lnf)));
          const bool acc = f_lt_ff(logu_s[q], ratio);
          if (acc) {
            held = s0 + si;
            lp = lpp;
            lnf = lnfp;
          }
          held_s[q] = held * 2 + (acc ? 1 : 0);
          lp_s[q] = lp;
          if ((s0 + si) % a.thin == 0) {
            rec[tid] = held;
            rec_lp[tid] = lp;
          }
        }
        cur_lp[tid] = lp;
        cur_lnf[tid] = lnf;
        cur[tid] = held;
      }
      __syncthreads();
      for (int i = gib; i < items; i += gpb) {
        const int ci = i / ns, si = i - ci * ns, s = s0 + si;
        if (s % a.thin != 0) continue;
        const int64_t c = c0 + ci, orow = c * a.buf_len + a.start + s / a.thin;
        const int h = held_s[ci * pitch + si], held = h >> 1;
        const float* src = held < 0 ? a.x0 + c * d : a.props + (c * a.S + held) * d;
        float* dst = a.out_pos + orow * d;
        if (a.vec) {
          for (int j = 4 * gl; j < d; j += 4 * G)
            __stcs(reinterpret_cast<float4*>(dst + j), __ldg(reinterpret_cast<const float4*>(src + j)));
        } else {
          for (int j = gl; j < d; j += G) __stcs(dst + j, __ldg(src + j));
        }
        if (gl == 0) {
          __stcs(a.out_logp + orow, lp_s[ci * pitch + si]);
          __stcs(a.out_acc + orow, (h & 1) ? 1.f : 0.f);
        }
      }
      __syncthreads();
    }
    for (int i = gib; i < nb; i += gpb) {
      const int64_t c = c0 + i;
      const float* src = rec[i] < 0 ? a.x0 + c * d : a.props + (c * a.S + rec[i]) * d;
      for (int j = gl; j < d; j += G) a.x_last[c * d + j] = __ldg(src + j);
      if (gl == 0 && a.lp_last) a.lp_last[c] = rec_lp[i];
    }
  }
}

// The scan for launches with enough chains to hide its latency: a lane group walks
// its chain's steps one after the other, evaluating each proposal as it comes and
// keeping the held position in registers, so that every proposal is read once
// and nothing is staged. Same bits as k_nf_accept.
template <int TGT, int G, int V>
__global__ void __launch_bounds__(256) k_nf_walk(const NfArgs a) {
  extern __shared__ __align__(16) float smem[];
  const int gl = threadIdx.x % G, gib = threadIdx.x / G, gpb = blockDim.x / G, gpw = 32 / G;
  const int d = a.d;
  float* stage = nullptr;
  const TargetConst<TGT> tc(a.tgt);
  if constexpr (TGT == FMC_TARGET_DENSE_GAUSSIAN) {
    stage = smem + gib * d;
  } else if constexpr (TGT == FMC_TARGET_DIAG_GAUSSIAN || TGT == FMC_TARGET_GAUSS_MIXTURE) {
    if (a.tab_smem) {
      stage_target_table<G, V>(a.tgt, smem);
      __syncthreads();
      stage = smem;
    }
  }
  const Rng rng = a.rng.at_epoch();
  const int64_t c_pad = ((int64_t)a.C + gpw - 1) / gpw * gpw;   // whole warps (the evaluations shuffle)
  for (int64_t c = (int64_t)blockIdx.x * gpb + gib; c < c_pad; c += (int64_t)gridDim.x * gpb) {
    const bool active = c < a.C;
    const int64_t cc = active ? c : 0;
    float x[V], g[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int j = gl * V + v;
      x[v] = (j < d) ? __ldg(a.x0 + cc * d + j) : 0.f;
    }
    float lp = target_eval<TGT, G, V, false>(a.tgt, tc, x, g, gl, stage);   // take_steps.py:201-203
    float lnf = __ldg(a.lnf + (int64_t)a.C * a.S + cc);
    float xr[V], lpr = lp;
#pragma unroll
    for (int v = 0; v < V; ++v) xr[v] = x[v];
    for (int s = 0; s < a.S; ++s) {
      const int64_t row = cc * a.S + s;
      float p[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int j = gl * V + v;
        p[v] = (j < d) ? __ldg(a.props + row * d + j) : 0.f;
      }
      const float lpp = target_eval<TGT, G, V, false>(a.tgt, tc, p, g, gl, stage);
      const float lnfp = __ldg(a.lnf + row);
      const float u = a.unif ? __ldg(a.unif + row) : u32_to_unit(rng.draw(cc, s, 0u, RNG_TAG_NF_UNIFORM).x);
      // ratio = (lp_p - lp_c) - (lnf_p - lnf_c)   (NF_proposal.py:102-104)
      const ff ratio = ff_add(two_sum(lpp, -lp), ff_neg(two_sum(lnfp, -lnf)));
      const bool acc = f_lt_ff(logf(u), ratio);
      if (acc) {
#pragma unroll
        for (int v = 0; v < V; ++v) x[v] = p[v];
        lp = lpp;
        lnf = lnfp;
      }
      if (s % a.thin == 0) {
        if (active) {
          const int64_t orow = cc * a.buf_len + a.start + s / a.thin;
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int j = gl * V + v;
            if (j < d) __stcs(a.out_pos + orow * d + j, x[v]);
          }
          if (gl == 0) {
            __stcs(a.out_logp + orow, lp);
            __stcs(a.out_acc + orow, acc ? 1.f : 0.f);
          }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) xr[v] = x[v];
        lpr = lp;
      }
    }
    if (active) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int j = gl * V + v;
        if (j < d) a.x_last[cc * d + j] = xr[v];
      }
      if (gl == 0 && a.lp_last) a.lp_last[cc] = lpr;
    }
  }
}

template <int TGT, int G, int V>
static int launch_nf_t(const NfArgs& a0, cudaStream_t st) {
  NfArgs a = a0;
  const int threads = 256, gpb = threads / G;
  // Chains of a block of k_nf_accept: enough to give every SM eight blocks (four of
  // the dense Gaussian's, which fill its registers), in whole rounds of them, with at most 512 proposals a round and no more chains than the
  // scan has threads; where a chain has few steps, at least one proposal per group.
  a.round_steps = a.S < kNfSteps ? a.S : kNfSteps;
  {
    const int64_t slots = (TGT == FMC_TARGET_DENSE_GAUSSIAN ? 4 : 8) * (int64_t)sm_count(), most = std::max(512 / a.round_steps, 1);
    const int64_t rounds = (a.C + most * slots - 1) / (most * slots);
    int64_t cb = (a.C + slots * rounds - 1) / (slots * rounds);
    cb = std::min<int64_t>(std::max<int64_t>(cb, gpb / a.round_steps), threads);
    a.chains_per_block = (int)std::max<int64_t>(cb, 1);
  }
  size_t floats = (TGT == FMC_TARGET_DENSE_GAUSSIAN) ? (size_t)gpb * a.d : 0;
  a.tab_smem = 0;
  if (TGT == FMC_TARGET_DIAG_GAUSSIAN || TGT == FMC_TARGET_GAUSS_MIXTURE) {
    const int tab = target_table_floats(TGT == FMC_TARGET_GAUSS_MIXTURE ? a.tgt.n_comp : 1, G * V);
    if (tab <= 33 * 256) {
      floats = tab;
      a.tab_smem = 1;
    }
  }
  floats = (floats + 3) / 4 * 4;
  a.scan_off = (int)floats;
  // From 20 warps of chains per SM on the walk's latency is hidden, and it reads the
  // proposals once: over 21 targets of 3 to 200 dims and 1 to 200 steps the staged
  // scan takes 1.0 to 1.5 of its time at 27 warps, up to 2.0 beyond, and 0.1 to 0.5
  // of it for 1000 chains of 30 steps. At 13 warps it takes 0.9 to 1.4 of it up to 16
  // steps or 8 dims, 0.6 to 1.05 otherwise. A single step has nothing to evaluate
  // ahead. Without the walk, 65,536 chains of the 5-D dual moon took, for 1
  // and 10 steps, 84 and 172 us, with it 15 and 64; 16,384 chains of a 64-D dense
  // Gaussian, 1 step: 158, with it 50.
  const double warps = (double)a.C * G / 32 / sm_count();
  const bool walk = a.S == 1 || warps >= 20.0 || (warps >= 10.0 && (a.S <= 16 || a.d <= 8));
  if (!walk) floats += (size_t)a.chains_per_block * (4 * (a.round_steps | 1) + 5);
  a.vec = a.d % 4 == 0 && ((uintptr_t)a.out_pos & 15) == 0 && ((uintptr_t)a.props & 15) == 0 &&
          ((uintptr_t)a.x0 & 15) == 0;
  const int per_block = walk ? gpb : a.chains_per_block;
  int64_t blocks = (a.C + per_block - 1) / per_block;
  const int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  auto kern = walk ? k_nf_walk<TGT, G, V> : k_nf_accept<TGT, G, V>;
  const size_t smem = floats * sizeof(float);
  FMC_CUDA_TRY(allow_smem(kern, smem));
  // proposals and their flow densities read, thinned rows written
  const double n_rec = (double)((a.S + a.thin - 1) / a.thin);
  KernelTimer kt(FMC_KT_NF_ACCEPT, st, 0.0,
                 (double)a.C * a.S * (4.0 * a.d + 4.0) + (double)a.C * n_rec * (4.0 * a.d + 8.0));
  kern<<<(int)blocks, threads, smem, st>>>(a);
  FMC_LAUNCH_CHECK();
  return FMC_OK;
}

template <int TGT>
static int launch_nf_tgt(const NfArgs& a, cudaStream_t st) {
  const int d = a.d;
#define NFC(g, v, lim) \
  if (d <= lim) return launch_nf_t<TGT, g, v>(a, st);
  NFC(4, 1, 4) NFC(8, 1, 8) NFC(8, 2, 16) NFC(8, 4, 32) NFC(16, 4, 64) NFC(32, 4, 128) NFC(32, 8, 256)
#undef NFC
  set_error("n_dim=%d too large for the global-step kernel", d);
  return FMC_ERR_UNSUPPORTED;
}

int check_target(const FmcTarget* t);

static size_t a256(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace fmc

using namespace fmc;

extern "C" int fmc_nf_workspace_size(const FmcFlow* flow, int32_t n_chains, int32_t n_steps, size_t* bytes) {
  FMC_CHECK_ARG(flow && bytes, "NULL pointer");
  FMC_CHECK_ARG(n_chains >= 1 && n_steps >= 1, "bad sizes");
  const int64_t rows = (int64_t)n_chains * n_steps;
  const int d = flow->n_dim;
  *bytes = a256((size_t)(rows + n_chains) * d * 4) + a256((size_t)(rows + n_chains) * 4) +
           flow_infer_ws_bytes(flow, rows + n_chains);
  return FMC_OK;
}

// the accept scan over precomputed proposals props [C * S, d] (row c * S + s)
// and flow log-densities lnf [C * S + C] (the proposals', then the current
// positions')
static int launch_accept(const FmcTarget* target, const float* x0, int32_t n_chains, int32_t n_steps,
                         int32_t thinning, uint64_t seed, uint64_t counter, const float* props, const float* lnf,
                         const float* unif, float* out_pos, float* out_logp, float* out_acc, int64_t buf_len,
                         int64_t cursor, float* x_last, float* lp_last, cudaStream_t st) {
  const int64_t n_rec = ((int64_t)n_steps + thinning - 1) / thinning;
  NfArgs a{};
  a.tgt = *target;
  a.x0 = x0;
  a.props = props;
  a.lnf = lnf;
  a.C = n_chains;
  a.d = target->n_dim;
  a.S = n_steps;
  a.thin = thinning;
  a.rng = Rng{(uint32_t)seed, (uint32_t)(seed >> 32), counter, rng_epoch()};
  a.unif = unif;
  a.out_pos = out_pos;
  a.out_logp = out_logp;
  a.out_acc = out_acc;
  a.buf_len = buf_len;
  a.start = cursor < buf_len - n_rec ? cursor : buf_len - n_rec;
  a.x_last = x_last;
  a.lp_last = lp_last;
  switch (target->kind) {
    case FMC_TARGET_DIAG_GAUSSIAN: return launch_nf_tgt<FMC_TARGET_DIAG_GAUSSIAN>(a, st);
    case FMC_TARGET_DUAL_MOON: return launch_nf_tgt<FMC_TARGET_DUAL_MOON>(a, st);
    case FMC_TARGET_GAUSS_MIXTURE: return launch_nf_tgt<FMC_TARGET_GAUSS_MIXTURE>(a, st);
    case FMC_TARGET_ROSENBROCK: return launch_nf_tgt<FMC_TARGET_ROSENBROCK>(a, st);
    default: return launch_nf_tgt<FMC_TARGET_DENSE_GAUSSIAN>(a, st);
  }
}

extern "C" int fmc_nf_global_steps(const FmcFlow* flow, const FmcTarget* target, const float* x0, int32_t n_chains,
                                   int32_t n_steps, int32_t thinning, uint64_t seed, uint64_t counter,
                                   const float* z, const float* unif, float* out_pos, float* out_logp,
                                   float* out_acc, int64_t buf_len, int64_t cursor, float* x_last, float* lp_last,
                                   void* ws, size_t ws_bytes, void* stream) {
  int rc = check_target(target);
  if (rc) return rc;
  FMC_CHECK_ARG(flow != nullptr, "flow is NULL");
  FMC_CHECK_ARG(flow->n_dim == target->n_dim, "flow n_dim %d != target n_dim %d", flow->n_dim, target->n_dim);
  FMC_CHECK_ARG(n_chains >= 0 && n_steps >= 1 && thinning >= 1, "bad sizes");
  const int64_t n_rec = ((int64_t)n_steps + thinning - 1) / thinning;
  FMC_CHECK_ARG(n_rec <= buf_len, "update of %lld rows does not fit a buffer of %lld rows", (long long)n_rec,
                (long long)buf_len);
  FMC_CHECK_ARG(cursor >= 0, "cursor < 0");
  if (n_chains == 0) return FMC_OK;
  FMC_CHECK_ARG(x0 && out_pos && out_logp && out_acc && x_last, "NULL array argument");
  size_t need = 0;
  if ((rc = fmc_nf_workspace_size(flow, n_chains, n_steps, &need))) return rc;
  FMC_CHECK_ARG(ws && ws_bytes >= need, "workspace of %zu bytes < %zu needed", ws_bytes, need);
  FMC_CHECK_ARG(((uintptr_t)ws & 255) == 0, "workspace must be 256-byte aligned");
  if (target->kind == FMC_TARGET_DENSE_GAUSSIAN)
    FMC_CHECK_SUPPORTED(target->n_dim <= 128, "dense Gaussian group kernel supports n_dim <= 128");
  cudaStream_t st = (cudaStream_t)stream;
  const int d = flow->n_dim;
  const int64_t rows = (int64_t)n_chains * n_steps;
  char* p = (char*)ws;
  float* props = (float*)p;  // [rows + C, d]: proposals, then the current positions
  p += a256((size_t)(rows + n_chains) * d * 4);
  float* lnf = (float*)p;
  p += a256((size_t)(rows + n_chains) * 4);
  void* fws = p;
  const size_t fws_bytes = ws_bytes - (size_t)(p - (char*)ws);

  if ((rc = flow_sample_rows(flow, seed, counter, z, rows, props, fws, fws_bytes, st))) return rc;
  FMC_CUDA_TRY(cudaMemcpyAsync(props + rows * d, x0, (size_t)n_chains * d * 4, cudaMemcpyDeviceToDevice, st));
  if ((rc = flow_apply_logprob(flow, props, rows + n_chains, lnf, fws, fws_bytes, st))) return rc;

  return launch_accept(target, x0, n_chains, n_steps, thinning, seed, counter, props, lnf, unif, out_pos, out_logp,
                       out_acc, buf_len, cursor, x_last, lp_last, st);
}

extern "C" int fmc_nf_accept(const FmcTarget* target, const float* x0, int32_t n_chains, int32_t n_steps,
                             int32_t thinning, uint64_t seed, uint64_t counter, const float* props, const float* lnf,
                             const float* unif, float* out_pos, float* out_logp, float* out_acc, int64_t buf_len,
                             int64_t cursor, float* x_last, float* lp_last, void* stream) {
  int rc = check_target(target);
  if (rc) return rc;
  FMC_CHECK_ARG(n_chains >= 0 && n_steps >= 1 && thinning >= 1, "bad sizes");
  const int64_t n_rec = ((int64_t)n_steps + thinning - 1) / thinning;
  FMC_CHECK_ARG(n_rec <= buf_len, "update of %lld rows does not fit a buffer of %lld rows", (long long)n_rec,
                (long long)buf_len);
  FMC_CHECK_ARG(cursor >= 0, "cursor < 0");
  if (n_chains == 0) return FMC_OK;
  FMC_CHECK_ARG(x0 && props && lnf && out_pos && out_logp && out_acc && x_last, "NULL array argument");
  if (target->kind == FMC_TARGET_DENSE_GAUSSIAN)
    FMC_CHECK_SUPPORTED(target->n_dim <= 128, "dense Gaussian group kernel supports n_dim <= 128");
  return launch_accept(target, x0, n_chains, n_steps, thinning, seed, counter, props, lnf, unif, out_pos, out_logp,
                       out_acc, buf_len, cursor, x_last, lp_last, (cudaStream_t)stream);
}
