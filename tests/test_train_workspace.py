"""Workspace of the flow losses' gradients: the activations kept for the
backward are bounded (beyond, they are recomputed layer by layer), a workspace
sized for one number of rows serves every smaller one, and the gradient is the
same with and without them. The CPU tests need the library's host arithmetic
only: a call without a workspace is refused with the bytes it needs."""
import ctypes
import re

import numpy as np
import pytest
import torch

from flowmc_gb300 import _lib, api

needs_lib = pytest.mark.skipif(not _lib.LIB_PATH.exists(), reason="libflowmc.so not built")
KEPT = 16 << 30


def _flow(d, L, hidden, nb, precision):
    s = _lib.FmcFlow()
    s.n_dim, s.n_layers, s.n_hidden, s.n_bins = d, L, len(hidden), nb
    for i, h in enumerate(hidden):
        s.hidden[i] = h
    s.range_min, s.range_max, s.min_bin_size, s.min_knot_slope = -10.0, 10.0, 1e-3, 1e-3
    s.precision = precision
    s.theta = s.aux = s.theta_bf16 = 256   # never read: the call is refused before
    return s


def _size(s, n):
    nb = ctypes.c_size_t()
    _lib.check(_lib.lib().fmc_flow_workspace_size(ctypes.byref(s), n, 1, ctypes.byref(nb)))
    return nb.value


def _least(s, n):
    """Fewest bytes that a gradient of n rows accepts."""
    assert _lib.lib().fmc_flow_loss_grad(ctypes.byref(s), 256, n, 256, 256, None, 0, None) != 0
    return int(re.search(r"< (\d+) needed", _lib.lib().fmc_last_error().decode()).group(1))


SHAPES = [(32, 8, [128, 128], 10, "FP32"), (64, 12, [128, 128], 16, "FP32"), (5, 4, [32, 32], 8, "FP32"),
          (32, 4, [256, 256], 10, "FP32"), (6, 1, [16], 4, "FP32"), (128, 12, [512, 512], 12, "BF16"),
          (64, 8, [256, 256], 8, "BF16")]


@needs_lib
@pytest.mark.parametrize("d,L,hidden,nb,prec", SHAPES)
def test_kept_activations_are_bounded(d, L, hidden, nb, prec):
    s = _flow(d, L, hidden, nb, getattr(_lib, f"PREC_{prec}"))
    P, H = 3 * nb + 8, -(-max(hidden) // 64) * 64
    for n in (1000, 16384, 200_000, 1_000_000, 4_000_000):
        # float32 rows of one layer: inputs of every layer, conditioner outputs and their gradients, hidden ones
        one_layer = 4 * n * ((L + 1) * d + 6 * d + 2 * (d // 2 + 1) * P + (len(hidden) + 2) * H + 64) + (256 << 20)
        assert _size(s, n) <= max(one_layer, KEPT + 4 * n * ((L + 1) * d + 64))


@needs_lib
@pytest.mark.parametrize("d,L,hidden,nb,prec", SHAPES)
def test_a_workspace_serves_every_smaller_batch(d, L, hidden, nb, prec):
    s = _flow(d, L, hidden, nb, getattr(_lib, f"PREC_{prec}"))
    rows = sorted({1, 63, 64, 255, 4864, 4865, 9727, 9728, 9729, 65536, 300_000, 4_000_000} |
                  {int(v) for v in np.exp(np.random.default_rng(d).uniform(0, np.log(4e6), 60))})
    for i, n in enumerate(rows):
        assert max(_least(s, m) for m in rows[:i + 1]) <= _size(s, n)


@pytest.mark.gpu
# FP32 in 16- and 64-row tiles; BF16 with and without x boxes and folded affines, below one 64-row block
@pytest.mark.parametrize("d,L,hidden,nb,prec,n", [(32, 8, [128, 128], 10, "float32", 1000), (5, 4, [32, 32], 8, "float32", 10000),
                                                  (33, 12, [64, 64, 64], 6, "float32", 333), (64, 4, [256, 256], 8, "bf16", 3000),
                                                  (128, 3, [512, 512], 12, "bf16", 1000), (7, 3, [64, 64], 8, "bf16", 200),
                                                  (8, 3, [64], 10, "bf16", 40)])
def test_gradient_without_kept_activations(cuda, d, L, hidden, nb, prec, n):
    """The same bits: every product, activation and sum over the batch keeps its
    order; only what is stored differs."""
    m = api.MaskedCouplingRQSpline(d, L, hidden, nb, api.PRNGKey(2), precision=prec, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(d + n)
    m.theta.add_(0.1 * torch.randn(m.theta.shape, generator=g, device="cuda"))
    m.sync_bf16()
    x = torch.randn(n, d, generator=g, device="cuda")
    loss, grad = (v.clone() for v in m.loss_and_grad(x))
    s = m.c_struct()
    least = _least(s, n)
    assert least < _size(s, n)
    ws = torch.full((least + 256,), 255, dtype=torch.uint8, device="cuda")   # NaN bit patterns
    p = ws.data_ptr() + (-ws.data_ptr()) % 256
    loss2, grad2 = torch.empty_like(loss), torch.empty_like(grad)
    _lib.check(_lib.lib().fmc_flow_loss_grad(ctypes.byref(s), x.data_ptr(), n, loss2.data_ptr(), grad2.data_ptr(), p,
                                             least, _lib.stream_handle(m.device)))
    assert torch.equal(loss, loss2)
    assert torch.equal(grad, grad2)
