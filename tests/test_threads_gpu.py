"""Threads that launch one kernel with different amounts of shared memory, each on
its own stream: a launch must not fail because another thread has just asked for
less, and every result is what the thread gets alone."""
import ctypes
import subprocess
import threading

import numpy as np
import pytest
import torch

from flowmc_gb300 import api
from flowmc_gb300 import build as B
from flowmc_gb300 import targets as TG
from flowmc_gb300.resource.kernel.base import run_local_steps

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"
__global__ void k_empty(int* out) {
  extern __shared__ int sm[];
  if (out != nullptr) *out = sm[0];
}
static int launch(size_t bytes) {
  k_empty<<<1, 32, bytes>>>(nullptr);
  return cudaGetLastError() | cudaDeviceSynchronize();
}
// one thread asks for 100 KB, another for 60, the first one launches: with the limit set
// to what each asks for, and with allow_smem
extern "C" __attribute__((visibility("default"))) int as_asked() {
  cudaFuncSetAttribute(k_empty, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
  cudaFuncSetAttribute(k_empty, cudaFuncAttributeMaxDynamicSharedMemorySize, 60 * 1024);
  return launch(100 * 1024);
}
extern "C" __attribute__((visibility("default"))) int allowed() {
  if (fmc::allow_smem(k_empty, 100 * 1024) || fmc::allow_smem(k_empty, 60 * 1024) || fmc::allow_smem(k_empty, 100)) return -1;
  return launch(100 * 1024);
}
"""


def test_a_smaller_request_leaves_a_larger_launch_alone(cuda, tmp_path):
    (tmp_path / "s.cu").write_text(SOURCE)
    subprocess.run([B.nvcc_path(), *B.NVCC_FLAGS, *B.ARCH, "-I", str(B.INCLUDE), "-I", str(B.CSRC), "-shared", "-o",
                    str(tmp_path / "s.so"), str(tmp_path / "s.cu")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "s.so"))
    assert lib.as_asked() != 0   # refused on the host: what a kernel's users must not do to one another
    assert lib.allowed() == 0


def _flow(d, hidden, rows, train):
    m = api.MaskedCouplingRQSpline(d, 3, hidden, 8, api.PRNGKey(1), device="cuda")
    x = torch.randn(rows, d, generator=torch.Generator(device="cuda").manual_seed(d), device="cuda")
    if train:
        return lambda: torch.cat([v.reshape(-1) for v in m.loss_and_grad(x)])
    return lambda: m.log_prob(x)


def _local(d, comps):
    C, S = 10000, 4
    tgt = TG.GaussianMixture(np.random.default_rng(d).normal(size=(comps, d)), 1.5)
    x0 = torch.randn(C, d, generator=torch.Generator(device="cuda").manual_seed(comps), device="cuda")
    kernel = api.MALA(0.05)

    def go():
        out = [torch.empty(s, device="cuda") for s in ((C, S, d), (C, S), (C, S))]
        run_local_steps(kernel, tgt, x0, S, 1, 5, 0, *out, 0)
        return out[0]
    return go


# the same kernel each (bins, row tile, direction; lanes and target), 54 to 120 KB of shared memory
@pytest.mark.parametrize("make", [lambda: [_flow(5, [32, 32], 40, False), _flow(32, [128, 128], 40, False)],
                                  lambda: [_flow(5, [32, 32], 40, True), _flow(32, [128, 128], 40, True)],
                                  lambda: [_local(250, 9), _local(250, 16)]], ids=["flow", "train", "local"])
def test_threads_with_different_shared_memory(cuda, make):
    calls = [f for _ in range(5) for f in make()]
    want = [f().clone() for f in calls]
    torch.cuda.synchronize()
    errors = []

    def work(f, w, repeats):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(repeats):
                    got = f()
                    if i % 100 == 0 and not torch.equal(got, w):
                        errors.append("differs")
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(f, w, 300)) for f, w in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
