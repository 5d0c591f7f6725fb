"""The forward that a RealNVP gradient keeps adds each product in the order of
its inputs, whatever the tile: a row's hidden activations, and with them the
relu derivatives, have the same bits in a small batch (64 x 32 tiles) and in a
large one (128-row tiles), so the gradient of a batch of copies of one row
set is that set's gradient to the rounding of its own sums."""
import numpy as np
import pytest
import torch

from test_realnvp import _random_model

pytestmark = pytest.mark.gpu


# float32 sums of n nearly equal parts: n 2^-24 at most, and far less in slices; 1e-5 of the largest entry
@pytest.mark.parametrize("d,L,H,n", [(32, 4, 256, 128), (7, 3, 64, 130), (13, 2, 100, 512)])
def test_gradient_of_repeated_rows(cuda, d, L, H, n):
    m = _random_model(d, L, H, 50 + d)
    x = torch.tensor(np.random.default_rng(3).normal(size=(n, d)), dtype=torch.float32, device="cuda")
    loss, grad = (v.clone() for v in m.loss_and_grad(x))
    many, gmany = m.loss_and_grad(x.repeat(64, 1))
    assert abs(float(many) - float(loss)) <= 1e-5 * max(1.0, abs(float(loss)))
    assert (gmany - grad).abs().max() <= 1e-5 * grad.abs().max()
