"""The ways through an FP32 flow pass: one fused launch in tiles of 16 or 64
rows, or the launches per layer. They give the same bits, so a row's results
do not depend on how many rows the call has; and wide flows, which a row tile
walks too slowly, keep the per-layer tiles."""
import pytest
import torch

from flowmc_gb300 import _lib, api

pytestmark = pytest.mark.gpu


def _flow(d, hidden, bins, layers=3):
    m = api.MaskedCouplingRQSpline(d, layers, hidden, bins, api.PRNGKey(1), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(d + bins)
    m.theta.add_(0.2 * torch.randn(m.theta.shape, generator=g, device="cuda"))
    return m, g


def _launches(f):
    n = _lib.launch_count()
    f()
    return _lib.launch_count() - n


# narrow, wide, one and three hidden layers, odd dimensions, more coordinates than one group
@pytest.mark.parametrize("d,hidden,bins", [(5, [32, 32], 8), (32, [128, 128], 10), (32, [512, 512], 10), (7, [400], 4),
                                           (33, [64, 200, 64], 5), (128, [16, 16], 4), (128, [768, 768], 12),
                                           (2, [8], 2)])
def test_a_row_has_the_same_bits_in_every_call(d, hidden, bins):
    m, g = _flow(d, hidden, bins)
    x = 3.0 * torch.randn(20003, d, generator=g, device="cuda")
    outs = lambda v: (m.log_prob(v), *m.forward(v), *m.inverse(v))
    whole = outs(x)
    for k in (1, 17, 300, 3000):
        for a, b in zip(outs(x[:k].contiguous()), whole):
            assert torch.equal(a, b[:k])
    s = m.sample(api.PRNGKey(3), 20003)
    assert torch.equal(m.sample(api.PRNGKey(3), 40), s[:40])


# the per-layer tiles were measured 1.4 to 5 times faster than a fused launch here
@pytest.mark.parametrize("d,hidden,bins,rows", [(32, [512, 512], 10, 100000), (32, [1024, 1024], 10, 100),
                                                (128, [768, 768], 12, 16), (128, [16, 16], 4, 65536),
                                                (8, [768, 768], 8, 20000)])
def test_slow_row_tiles_are_not_taken(d, hidden, bins, rows):
    m, g = _flow(d, hidden, bins)
    x = torch.randn(rows, d, generator=g, device="cuda")
    assert _launches(lambda: m.log_prob(x)) > 3


# and the fused launch 1.5 to 4 times faster here
@pytest.mark.parametrize("d,hidden,bins,rows", [(5, [32, 32], 8, 600), (32, [128, 128], 10, 100003),
                                                (8, [64, 64], 8, 5000), (32, [64, 64], 10, 9728)])
def test_fast_row_tiles_are_taken(d, hidden, bins, rows):
    m, g = _flow(d, hidden, bins)
    x = torch.randn(rows, d, generator=g, device="cuda")
    assert _launches(lambda: m.log_prob(x)) == 1
