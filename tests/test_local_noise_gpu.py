"""The noise of the local steps is the same whether a launch draws it in chunks of
four steps or each lane draws its own (launches of one, two, three, five ... steps
in more than 16 dimensions): the first steps of a long launch are those of a
short one, bit for bit."""
import numpy as np
import pytest
import torch

from flowmc_gb300 import api
from flowmc_gb300 import targets as TG
from flowmc_gb300.resource.kernel.base import run_local_steps

pytestmark = pytest.mark.gpu


def _run(kernel, tgt, x0, S):
    C, d = x0.shape
    out = [torch.full(s, -7.0, device="cuda") for s in ((C, S, d), (C, S), (C, S))]
    last = run_local_steps(kernel, tgt, x0, S, 1, 3, 1, *out, 0)
    return out, last


# lane shapes (8, 2), (8, 4), (16, 4), (32, 4), (32, 8); odd dimensions; 64- and 256-thread blocks
@pytest.mark.parametrize("kind,d,C", [("grw", 12, 33), ("mala", 17, 100), ("grw", 31, 60000), ("hmc", 64, 500),
                                      ("mala", 50, 30000), ("grw", 128, 20), ("mala", 101, 11000), ("hmc", 130, 77),
                                      ("grw", 250, 10000)])
@pytest.mark.parametrize("target", ["diag", "rosenbrock", "mixture"])
def test_short_launches_start_long_ones(cuda, kind, d, C, target):
    r = np.random.default_rng(d)
    tgt = {"diag": lambda: TG.DiagGaussian(d, mean=r.normal(size=d), inv_var=r.uniform(0.5, 2, d)),
           "rosenbrock": lambda: TG.Rosenbrock(d), "mixture": lambda: TG.GaussianMixture(r.normal(size=(3, d)), 1.5)}[target]()
    kernel = {"grw": lambda: api.GaussianRandomWalk(0.1), "mala": lambda: api.MALA(0.03),
              "hmc": lambda: api.HMC(1, 0.02, 3)}[kind]()
    x0 = 0.3 * torch.randn(C, d, generator=torch.Generator(device="cuda").manual_seed(d), device="cuda")
    (pos, lp, acc), _ = _run(kernel, tgt, x0, 16)   # whole chunks
    for S in (1, 2, 3, 4, 5, 6, 7, 9, 10, 11, 13):
        (p, l, a), (x_last, lp_last) = _run(kernel, tgt, x0, S)
        assert torch.equal(p, pos[:, :S]) and torch.equal(l, lp[:, :S]) and torch.equal(a, acc[:, :S])
        assert torch.equal(x_last, pos[:, S - 1])
