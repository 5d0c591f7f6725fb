"""Workspace of the RealNVP gradient: what a batch keeps is bounded (larger ones
run in chunks of rows), and a workspace sized for one number of rows serves every
smaller one. Host arithmetic only, apart from the test of a batch in chunks."""
import ctypes

import numpy as np
import pytest
import torch

from flowmc_gb300 import _lib
from flowmc_gb300.resource.model.nf_model.realNVP import FmcRealNVP
from test_realnvp import _random_model

needs_lib = pytest.mark.skipif(not _lib.LIB_PATH.exists(), reason="libflowmc.so not built")
KEPT = 16 << 30
SHAPES = [(32, 8, 256), (2, 2, 8), (64, 12, 512), (100, 4, 30)]


def _size(d, L, H, n):
    s = FmcRealNVP()
    s.n_dim, s.n_layers, s.n_hidden, s.dt = d, L, H, 1.0
    nb = ctypes.c_size_t()
    _lib.check(_lib.lib().fmc_rnvp_workspace_size(ctypes.byref(s), n, 1, ctypes.byref(nb)))
    return nb.value


@needs_lib
@pytest.mark.parametrize("d,L,H", SHAPES)
def test_kept_activations_are_bounded(d, L, H):
    for n in (1000, 100_000, 1_000_000, 4_000_000, 40_000_000):
        assert _size(d, L, H, n) <= KEPT + 4 * n + (1 << 28)   # log-densities; weights, slices and partial sums


@needs_lib
@pytest.mark.parametrize("d,L,H", SHAPES)
def test_a_workspace_serves_every_smaller_batch(d, L, H):
    rows = sorted({1, 255, 256, 257, 4864, 4865, 65536} |
                  {int(v) for v in np.exp(np.random.default_rng(d).uniform(0, np.log(4e6), 300))})
    sizes = [_size(d, L, H, n) for n in rows]
    assert sizes == sorted(sizes)


@pytest.mark.gpu
def test_gradient_in_chunks(cuda):
    """Two whole chunks: with twice the rows every product and sum of a chunk is half of
    what it is alone (an exact scaling), and the two gradients are added."""
    d, L, H = 16, 16, 1024
    lo, hi = 1, 1 << 12   # in 256 rows: the workspace grows by more than the log-densities up to one chunk
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if _size(d, L, H, 256 * mid) - _size(d, L, H, 256 * mid - 256) > 256 * 8 else (lo, mid)
    k = 256 * lo
    assert 60000 < k < 70000
    m = _random_model(d, L, H, 5)
    x = torch.tensor(np.random.default_rng(6).normal(size=(2 * k, d)), dtype=torch.float32, device="cuda")
    parts = [tuple(v.clone() for v in m.loss_and_grad(v)) for v in (x[:k], x[k:])]
    loss, grad = m.loss_and_grad(x)
    want = (float(parts[0][0]) + float(parts[1][0])) / 2
    assert abs(float(loss) - want) <= 1e-5 * max(1.0, abs(want))   # float32 mean of log-densities in another order
    assert torch.equal(grad, 0.5 * parts[0][1] + 0.5 * parts[1][1])
