"""FP32 training takes the fused passes where they are the faster way: nine
launches, whatever the layers, against some fifteen per layer."""
import pytest
import torch

from flowmc_gb300 import _lib, api

pytestmark = pytest.mark.gpu


# measured: fused 1.08 to 1.18 times the layers' time (many coordinates, narrow layers); 1.5 to 4 times faster
@pytest.mark.parametrize("d,hidden,bins,rows,fused", [(250, [48, 48], 16, 1000, False), (128, [16, 16], 16, 20000, False),
                                                      (200, [16], 16, 20000, False), (5, [32, 32], 8, 10000, True),
                                                      (32, [128, 128], 10, 16384, True), (8, [64], 4, 100, True)])
def test_the_faster_way_is_taken(cuda, d, hidden, bins, rows, fused):
    m = api.MaskedCouplingRQSpline(d, 4, hidden, bins, api.PRNGKey(1), device="cuda")
    x = torch.randn(rows, d, generator=torch.Generator(device="cuda").manual_seed(d), device="cuda")
    n = _lib.launch_count()
    m.loss_and_grad(x)
    assert (_lib.launch_count() - n < 15) == fused
