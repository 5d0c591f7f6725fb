"""A RealNVP row has the same bits in a call of one row and of many (the products
of the forward are added in the order of the inputs, whatever tile the number of
rows asks for), and the loss is that of log_prob."""
import numpy as np
import pytest
import torch

from flowmc_gb300 import api
from test_realnvp import _random_model

pytestmark = pytest.mark.gpu


# narrow and wide, odd sizes, outputs of more than 32 columns, few inputs
@pytest.mark.parametrize("d,L,H", [(32, 4, 256), (5, 3, 64), (13, 2, 100), (64, 2, 30), (2, 2, 8), (100, 2, 300)])
def test_a_row_has_the_same_bits_in_every_call(cuda, d, L, H):
    m = _random_model(d, L, H, 60 + d)
    n = 70000   # a chunk of 65,536 rows and a remainder
    x = torch.tensor(np.random.default_rng(4).normal(size=(n, d)), dtype=torch.float32, device="cuda")
    outs = lambda v: (m.log_prob(v), *m.forward(v), *m.inverse(v))
    whole = outs(x)
    for k in (1, 100, 3000):
        for a, b in zip(outs(x[:k].contiguous()), whole):
            assert torch.equal(a, b[:k])
    for a, b in zip(outs(x[65536:].contiguous()), whole):
        assert torch.equal(a, b[65536:])
    s = m.sample(api.PRNGKey(3), n)
    assert torch.equal(m.sample(api.PRNGKey(3), 40), s[:40])


@pytest.mark.parametrize("d,L,H", [(32, 4, 256), (13, 2, 100)])
def test_loss_of_one_row_is_its_log_prob(cuda, d, L, H):
    m = _random_model(d, L, H, 70 + d)
    for i in range(8):
        x = torch.tensor(np.random.default_rng(i).normal(size=(1, d)), dtype=torch.float32, device="cuda")
        assert float(m.loss_and_grad(x)[0]) == -float(m.log_prob(x)[0])
