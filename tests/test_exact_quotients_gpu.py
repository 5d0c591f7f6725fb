"""The quotients that replace the division operator (common.cuh: MarkDiv,
ConstDiv; spline.cuh: softmax_div) have the operator's bits over the ranges that
their users check, and the targets built on them (targets.cuh) the bits that
they have with the operator. A kernel compiled here compares them."""
import ctypes
import subprocess

import numpy as np
import pytest
import torch

from flowmc_gb300 import build as B

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "spline.cuh"
#include "targets.cuh"
using namespace fmc;
__device__ bool same(float p, float q) { return __float_as_uint(p) == __float_as_uint(q) || (p != p && q != q); }

// bad[0]: MarkDiv, bad[1]: two() where the divisor's significand is even, bad[2]: numerators compared with two()
__global__ void k_quot(const float* b, const float* a, int64_t na, unsigned long long* bad) {
  const ConstDiv by(b[blockIdx.y]);
  if (!by.in_range) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < na; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = a[(int64_t)blockIdx.y * na + i], q = __fdiv_rn(x, by.b);
    if (!same(by(x), q)) atomicAdd(bad, 1ull);
    if (by.even) {
      atomicAdd(bad + 2, 1ull);
      if (!same(by.two(x), q)) atomicAdd(bad + 1, 1ull);
    }
  }
}
template <int K>
__global__ void k_softmax(const float* r, int64_t n, unsigned long long* bad) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float p[K], q[K];
  const float s = softmax_num<K>(r + i * K, p);
  for (int k = 0; k < K; ++k) q[k] = __fdiv_rn(p[k], s);
  softmax_div<K>(p, s);
  for (int k = 0; k < K; ++k)
    if (!same(p[k], q[k])) atomicAdd(bad, 1ull);
}
template <typename C> __device__ void operators(C&);
template <> __device__ void operators(TargetConst<FMC_TARGET_DUAL_MOON>& c) { c.fast = false; }
template <> __device__ void operators(TargetConst<FMC_TARGET_ROSENBROCK>& c) { c.fast = 0; }
// value and gradient of d <= 8 coordinates with the target's constants and with the operator
template <int TGT>
__global__ void k_target(const FmcTarget t, const float* x, int64_t n, unsigned long long* bad) {
  const int gl = threadIdx.x % 4;
  const int64_t i = blockIdx.x * (int64_t)(blockDim.x / 4) + threadIdx.x / 4;   // n: whole blocks
  float v[2], g[2], h[2];
  for (int u = 0; u < 2; ++u) v[u] = gl * 2 + u < t.n_dim ? x[i * t.n_dim + gl * 2 + u] : 0.f;
  TargetConst<TGT> tc(t), op(t);
  operators(op);
  const float lp = target_eval<TGT, 4, 2, true>(t, tc, v, g, gl, nullptr);
  const float lq = target_eval<TGT, 4, 2, true>(t, op, v, h, gl, nullptr);
  if (!same(lp, lq)) atomicAdd(bad, 1ull);
  for (int u = 0; u < 2; ++u)
    if (gl * 2 + u < t.n_dim && !same(g[u], h[u])) atomicAdd(bad, 1ull);
}
#define OUT extern "C" __attribute__((visibility("default"))) int
OUT quot(const float* b, int nb, const float* a, int64_t na, unsigned long long* bad) {
  k_quot<<<dim3(64, nb), 256>>>(b, a, na, bad);
  return cudaDeviceSynchronize();
}
OUT softmax8(const float* r, int64_t n, unsigned long long* bad) {
  k_softmax<8><<<(unsigned)((n + 255) / 256), 256>>>(r, n, bad);
  return cudaDeviceSynchronize();
}
OUT target(int kind, int d, const float* scalars, const float* x, int64_t n, unsigned long long* bad) {
  FmcTarget t{};
  t.kind = kind;
  t.n_dim = d;
  for (int i = 0; i < 4; ++i) t.scalars[i] = scalars[i];
  if (kind == FMC_TARGET_DUAL_MOON) k_target<FMC_TARGET_DUAL_MOON><<<(unsigned)(n / 64), 256>>>(t, x, n, bad);
  else k_target<FMC_TARGET_ROSENBROCK><<<(unsigned)(n / 64), 256>>>(t, x, n, bad);
  return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(SOURCE)
    subprocess.run([B.nvcc_path(), *B.NVCC_FLAGS, *B.ARCH, "-I", str(B.INCLUDE), "-I", str(B.CSRC), "-shared", "-o",
                    str(d / "q.so"), str(d / "q.cu")], check=True)
    return ctypes.CDLL(str(d / "q.so"))


def _floats(rng, n, lo, hi):
    """Random signs and significands, exponents lo .. hi - 1, with some extreme significands."""
    m = rng.integers(0, 1 << 23, n, dtype=np.uint32)
    m[:: 17] = 0x7FFFFF
    m[5:: 17] = 0
    m[9:: 17] = 1
    e = rng.integers(lo, hi, n).astype(np.int64) + 127
    s = rng.integers(0, 2, n, dtype=np.uint32)
    return ((s << 31) | (e.astype(np.uint32) << 23) | m).view(np.float32)


def _count(n=1):
    return torch.zeros(n, dtype=torch.int64, device="cuda")


def test_quotients_have_the_operators_bits(lib):
    rng = np.random.default_rng(0)
    b = np.concatenate([_floats(rng, 160, -30, 30), rng.uniform(1, 16, 60).astype(np.float32),
                        np.float32([2.0 ** -30, 2.0 ** 30, -2.0 ** 30, 20.0, 10.0, 0.1, 0.6, 1.0, 3.0, 16.0])])
    na = 100_000
    a = np.empty((len(b), na), np.float32)
    for i, v in enumerate(b):
        far = _floats(rng, na // 2, -60, 60)
        # numerators whose quotient lies next to a midpoint of two floats: one ulp about b (q + ulp(q) / 2)
        q = np.abs(_floats(rng, na - na // 2, -20, 20))
        near = (v.astype(np.float64) * (q.astype(np.float64) + np.spacing(q).astype(np.float64) / 2)).astype(np.float32)
        step = rng.integers(-1, 2, near.size)
        near = np.where(step < 0, np.nextafter(near, np.float32(-3e38)), np.where(step > 0, np.nextafter(near, np.float32(3e38)), near))
        a[i] = np.concatenate([far, near])
    a[:, :4] = np.float32([2.0 ** -60, 2.0 ** 60, -2.0 ** 60, -2.0 ** -60])
    tb, ta, bad = torch.tensor(b, device="cuda"), torch.tensor(a, device="cuda"), _count(3)
    assert lib.quot(ctypes.c_void_p(tb.data_ptr()), len(b), ctypes.c_void_p(ta.data_ptr()), ctypes.c_int64(na),
                    ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad[:2].tolist() == [0, 0]
    assert bad[2].item() > 20 * na   # even significands were among the divisors


# spreads that keep every numerator above 2^-60, cross it, and leave the float range
@pytest.mark.parametrize("spread", [1.0, 8.0, 25.0, 42.0, 200.0])
def test_softmax_has_the_operators_bits(lib, spread):
    r = torch.tensor(np.random.default_rng(1).uniform(-spread, spread, (1 << 20, 8)), dtype=torch.float32, device="cuda")
    r[:4] = torch.tensor([[-3e38] * 8, [0.0] * 8, [0.0] * 7 + [float("nan")], [float("-inf")] + [0.0] * 7], device="cuda")
    bad = _count()
    assert lib.softmax8(ctypes.c_void_p(r.data_ptr()), ctypes.c_int64(r.shape[0]), ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0


# divisors with even and odd significands, at the ends of the checked range and outside it
@pytest.mark.parametrize("kind,d", [("moon", 5), ("rosenbrock", 8), ("rosenbrock", 7)])
@pytest.mark.parametrize("div", [20.0, 0.1, 3.0, 0.6, 2.0 ** -30, 2.0 ** 30, 1.9999999, 2.0 ** -31, 3e31, 1e-38])
def test_targets_have_the_operators_bits(lib, kind, d, div):
    rng = np.random.default_rng(2)
    n = 1 << 16
    x = (rng.normal(size=(n, d)) * np.exp(rng.uniform(-3, 3, (n, 1)))).astype(np.float32)
    x[: n // 4] = _floats(rng, (n // 4) * d, -45, 45).reshape(-1, d)   # outside the checked numerators as well
    x[:3] = [[1.0] * d, [0.0] * d, [float("inf")] * d]
    scalars = {"moon": [2.0, div, 3.0, 1.7 * div if div < 1e30 else div], "rosenbrock": [div, 1.0, 5.0, 0.0]}[kind]
    code = {"moon": 1, "rosenbrock": 3}[kind]
    tx, bad = torch.tensor(x, device="cuda"), _count()
    assert lib.target(code, d, (ctypes.c_float * 4)(*scalars), ctypes.c_void_p(tx.data_ptr()), ctypes.c_int64(n),
                      ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0
