"""The two accept kernels of the global step, the staged scan and the walk by
lane groups, give the same chains: a chain's accepts depend on its own row,
proposals and random numbers only, so the first chains of a call with many
(walked) equal those of a call with few (scanned), bit for bit; and so do the
first steps of a long call and a call of one step, which is walked whatever
the number of chains."""
import ctypes

import numpy as np
import pytest
import torch

from flowmc_gb300 import _lib
from flowmc_gb300 import targets as TG

pytestmark = pytest.mark.gpu


def _target(kind, d):
    r = np.random.default_rng(d)
    return {"moon": lambda: TG.DualMoon(d), "rosenbrock": lambda: TG.Rosenbrock(d),
            "diag": lambda: TG.DiagGaussian(d, mean=r.normal(size=d), inv_var=r.uniform(0.5, 2, d)),
            "mixture": lambda: TG.GaussianMixture(r.normal(size=(5, d)), 1.5),
            "dense": lambda: TG.DenseGaussian(np.eye(d) + 0.1 * np.ones((d, d)))}[kind]()


def _accept(tgt, x0, props, lnf, thin, unif=None):
    C, S, d = props.shape
    rows = -(-S // thin)
    out = [torch.full(s, -7.0, device="cuda") for s in ((C, rows, d), (C, rows), (C, rows), (C, d), (C,))]
    pos, lp, acc, x_last, lp_last = out
    s = tgt.c_struct()
    _lib.check(_lib.lib().fmc_nf_accept(
        ctypes.byref(s), x0.data_ptr(), C, S, thin, 11, 3, props.data_ptr(), lnf.data_ptr(),
        None if unif is None else unif.data_ptr(), pos.data_ptr(), lp.data_ptr(), acc.data_ptr(), rows, 0,
        x_last.data_ptr(), lp_last.data_ptr(), _lib.stream_handle(x0.device)))
    return out


def _inputs(d, C, S):
    g = torch.Generator(device="cuda").manual_seed(d * 1000 + S)
    x0 = torch.randn(C, d, generator=g, device="cuda")
    props = torch.randn(C, S, d, generator=g, device="cuda")
    lnf = -0.5 * (torch.cat([props.reshape(-1, d), x0]) ** 2).sum(1)   # like a flow's densities: some accepts, some not
    unif = torch.rand(C, S, generator=g, device="cuda").clamp_min(1e-6)
    return x0, props, lnf, unif


def _first(props, lnf, k):
    C, S, _ = props.shape
    return torch.cat([lnf[:C * S].view(C, S)[:k].reshape(-1), lnf[C * S:C * S + k]])


# lane groups of 4, 8, 16 and 32, odd rows, thinning, a round and a part, explicit uniforms
@pytest.mark.parametrize("kind,d,S,thin,explicit", [("moon", 3, 2, 1, False), ("moon", 5, 7, 2, True),
                                                    ("diag", 8, 65, 1, False), ("mixture", 20, 3, 1, False),
                                                    ("dense", 33, 5, 3, True), ("rosenbrock", 64, 4, 1, False),
                                                    ("rosenbrock", 130, 2, 1, False)])
def test_walked_and_scanned_chains_agree(kind, d, S, thin, explicit):
    G = 4 if d <= 4 else 8 if d <= 32 else 16 if d <= 64 else 32
    C = 20 * 32 * torch.cuda.get_device_properties(0).multi_processor_count // G   # walked whatever the steps
    tgt = _target(kind, d)
    x0, props, lnf, unif = _inputs(d, C, S)
    u = unif if explicit else None
    many = _accept(tgt, x0, props, lnf, thin, u)
    for k in (C - 1, 300, 17, 1):
        few = _accept(tgt, x0[:k].contiguous(), props[:k].contiguous(), _first(props, lnf, k), thin,
                      None if u is None else u[:k].contiguous())
        for a, b in zip(few, many):
            assert torch.equal(a, b[:k])
    assert 0.02 < many[2].mean().item() < 0.98   # both outcomes occur


@pytest.mark.parametrize("kind,d,C", [("moon", 5, 100), ("mixture", 64, 33), ("dense", 7, 1)])
def test_one_step_is_the_first_of_many(kind, d, C):
    tgt = _target(kind, d)
    x0, props, lnf, _ = _inputs(d, C, 9)
    long = _accept(tgt, x0, props, lnf, 1)
    one = _accept(tgt, x0, props[:, :1].contiguous(), torch.cat([lnf[:C * 9].view(C, 9)[:, 0], lnf[C * 9:]]), 1)
    for a, b in zip(one[:3], long[:3]):
        assert torch.equal(a, b[:, :1])
