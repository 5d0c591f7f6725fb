"""Edges of the kernels' tiles, groups and dispatch lines against the oracle:
row counts beside the 16- and 64-row tiles of the fused FP32 flow passes and
the line between them, widths on both sides of what they take, coordinate
groups of the tensor-core spline kernels that end part empty, the RealNVP
product's tile shapes, the NF accept scan's 64-step rounds, the local kernel's
block shapes and divisors, and the batched sampler's packed positions.

Tolerances are those of the same quantities elsewhere in this suite: FP32
flow values and gradients 1e-4 (gradients of the largest entry), BF16 values
within three times what bfloat16 operands alone cause, BF16 losses 2e-2 with
the gradient's cosine above 0.999, RealNVP 1e-4, positions and
log-densities of a trajectory 1e-4 where no accept decision is a tie. Where
two routes compute the same thing the bits are equal.
"""
import numpy as np
import pytest
import torch

from oracle import flow_torch as FT
from oracle import kernels as K
from oracle import realnvp as R
from test_flow_bf16_deep_gpu import assert_within_bf16, bf16_flow
from test_flow_gpu import gpu_grad_to_full, gpu_model, rand_flow, to_f32
from test_realnvp import _oracle_of, _random_model

pytestmark = pytest.mark.gpu


def _tall():
    """The first row count that the fused FP32 passes take in 64-row tiles."""
    return 64 * torch.cuda.get_device_properties(0).multi_processor_count


FLOWS = [(5, 2, (24,), 6), (7, 3, (9, 11), 4), (66, 2, (50, 70), 8), (6, 2, (17, 17, 17, 17), 10),
         (4, 2, (1000,), 5)]   # the last: wider than the fused pass takes


@pytest.mark.parametrize("d,L,hidden,nb", FLOWS)
def test_fp32_flow_pass_row_edges(cuda, d, L, hidden, nb):
    fl = to_f32(rand_flow(d, L, hidden, nb, seed=d + nb))
    m = gpu_model(fl, hidden)
    rng = np.random.default_rng(3)
    for n in (1, 15, 16, 17, 63, 65, _tall() - 1, _tall() + 1):
        x = (rng.normal(size=(n, d)) * 2.5).astype(np.float32)
        xt = torch.tensor(x, device="cuda")
        k = np.unique(np.r_[:min(n, 20), max(n - 70, 0):n])   # rows compared
        x64 = x[k].astype(np.float64)
        (y, ld), (xi, ldi) = m.forward(xt), m.inverse(xt)
        for got, want in ((y, fl.forward(x64)[0]), (xi, fl.inverse(x64)[0])):
            np.testing.assert_allclose(got.cpu().numpy()[k], want, rtol=1e-4, atol=1e-4)
        for got, want in ((ld, fl.forward(x64)[1]), (ldi, fl.inverse(x64)[1]), (m.log_prob(xt), fl.log_prob(x64))):
            np.testing.assert_allclose(got.cpu().numpy()[k], want, rtol=1e-4, atol=1e-4 * max(1, np.abs(want).max()))


@pytest.mark.parametrize("d,L,hidden,nb", [(5, 4, (32, 32), 8), (7, 3, (24,), 5), (9, 2, (17, 20, 33), 6),
                                           (6, 2, (136, 40), 8)])   # the last: wider than the fused gradient takes
def test_fp32_flow_gradient_row_edges(cuda, d, L, hidden, nb):
    fl = to_f32(rand_flow(d, L, hidden, nb, seed=40 + d))
    m = gpu_model(fl, hidden)
    rng = np.random.default_rng(5)
    for n in (1, 15, 17, 63, 65, _tall() + 1):
        x = (rng.normal(size=(n, d)) * 2).astype(np.float32)
        loss, grad = m.loss_and_grad(torch.tensor(x, device="cuda"))
        oloss, og = FT.loss_and_grad(fl, x.astype(np.float64))
        assert abs(loss.item() - oloss) <= 1e-4 * max(1, abs(oloss))
        np.testing.assert_allclose(gpu_grad_to_full(m, grad), og, atol=1e-4 * np.abs(og).max(), rtol=0)


# x boxes of 2, 4, 5 and 3 chunks per row with a last group of 4, 2, 2 and 2
# coordinates, two row strides that no box takes, deep input gradients (on CTA pairs)
@pytest.mark.parametrize("d,L,hidden,nb,n", [(8, 3, (64, 64), 16, 129), (20, 3, (64, 128), 8, 500),
                                             (24, 3, (72,), 6, 1000), (16, 2, (128, 128), 12, 4001),
                                             (18, 2, (64, 64), 8, 300), (15, 3, (64, 64), 12, 129),
                                             (56, 2, (512, 512), 12, 10000)])
def test_bf16_flow_group_edges(cuda, d, L, hidden, nb, n):
    from flowmc_gb300 import _lib
    fl = to_f32(rand_flow(d, L, hidden, nb, seed=60 + d, wscale=0.3))
    m = gpu_model(fl, hidden, precision="bf16")
    x = (np.random.default_rng(6).normal(size=(n, d)) * 1.5).astype(np.float32)
    xt = torch.tensor(x, device="cuda")
    k = np.unique(np.r_[:min(n, 150), max(n - 150, 0):n])
    x64 = x[k].astype(np.float64)
    fb = bf16_flow(fl)
    for got, want, emul, what in ((m.forward(xt), fl.forward(x64), fb.forward(x64), "forward"),
                                  (m.inverse(xt), fl.inverse(x64), fb.inverse(x64), "inverse")):
        for i in (0, 1):
            assert_within_bf16(got[i].cpu().numpy()[k], want[i], emul[i], what)
    loss, grad = m.loss_and_grad(xt)
    assert _lib.device_error() == 0
    oloss, og = FT.loss_and_grad(fl, x.astype(np.float64))
    assert abs(loss.item() - oloss) <= 2e-2 * max(1, abs(oloss))
    gg = gpu_grad_to_full(m, grad)
    assert float(gg @ og / (np.linalg.norm(gg) * np.linalg.norm(og))) > 0.999
    # the training forward runs the layers' kernels as log_prob does
    assert loss.item() == pytest.approx(-m.log_prob(xt).mean().item(), rel=1e-5, abs=1e-5)


@pytest.mark.parametrize("d,L,H,n", [(33, 2, 64, 1), (7, 3, 30, 100), (64, 2, 100, 4097), (16, 4, 130, 20001)])
def test_realnvp_tile_edges(cuda, d, L, H, n):
    m = _random_model(d, L, H, 20 + d)
    o = _oracle_of(m)
    x = np.random.default_rng(7).normal(size=(n, d))
    xt = torch.tensor(x, dtype=torch.float32, device="cuda")
    x = xt.cpu().numpy().astype(np.float64)
    np.testing.assert_allclose(m.log_prob(xt).cpu().numpy(), o.log_prob(x), rtol=1e-4, atol=1e-3)
    loss, grad = m.loss_and_grad(xt)
    lo, go = R.loss_and_grad(o, x)
    want = R.pack(go, L)
    assert abs(float(loss) - lo) < 1e-4 * max(1.0, abs(lo))
    assert np.abs(grad.cpu().numpy() - want).max() < 1e-4 * np.abs(want).max()


# rounds of 64 steps, several chains per block, rows that are not whole 16-byte words
@pytest.mark.parametrize("d,C,S,thin", [(2, 3, 1, 1), (5, 9, 64, 1), (5, 9, 65, 3), (8, 4, 130, 2), (3, 1300, 3, 1)])
def test_nf_accept_step_edges(cuda, d, C, S, thin):
    from flowmc_gb300 import targets as TG
    from flowmc_gb300.resource.kernel.NF_proposal import NFProposal
    fl = to_f32(rand_flow(d, 2, (16,), 6, seed=80 + d, wscale=0.2))
    m = gpu_model(fl, (16,))
    tgt = TG.GaussianMixture(np.random.default_rng(1).normal(size=(3, d)), 1.5)
    rng = np.random.default_rng(9)
    x0 = rng.normal(size=(C, d)).astype(np.float32)
    z = rng.normal(size=(C, S, d)).astype(np.float32)
    u = rng.uniform(1e-6, 1, size=(C, S)).astype(np.float32)
    rows = -(-S // thin)
    pos, lp, acc = (torch.full(s, -np.inf, device="cuda") for s in ((C, rows, d), (C, rows), (C, rows)))
    up = lambda a: torch.tensor(a, device="cuda")
    NFProposal(m).group_steps(9, up(x0), tgt, S, thin, pos, lp, acc, 0, noise=up(z), uniform=up(u))
    ox, olp, oacc = K.nf_proposal_kernel(fl, tgt.describe(), x0.astype(np.float64), z.astype(np.float64),
                                         u.astype(np.float64))
    acc = acc.cpu().numpy()
    ok = (acc == oacc[:, ::thin]).all(1)   # chains without a tie flip
    assert ok.mean() >= 0.95
    np.testing.assert_allclose(pos.cpu().numpy()[ok], ox[:, ::thin][ok], rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(lp.cpu().numpy()[ok], olp[:, ::thin][ok], rtol=1e-4, atol=1e-3)


def _local(tgt, kind, x0, S, thin, noise=None, unif=None):
    from flowmc_gb300.resource.kernel.base import run_local_steps
    from test_local_gpu import _kernel
    C, d = x0.shape
    rows = -(-S // thin)
    out = [torch.full(s, -np.inf, device="cuda") for s in ((C, rows, d), (C, rows), (C, rows))]
    run_local_steps(_kernel(kind, 0.05, 3), tgt, x0, S, thin, 77, 0, *out, 0, noise=noise, uniform=unif)
    return out


@pytest.mark.parametrize("kind", ["mala", "hmc", "grw"])
@pytest.mark.parametrize("name,d", [("dual", 5), ("rosen", 12), ("mix", 9), ("mix", 64), ("diag", 33)])
def test_block_shape_does_not_change_a_chain(cuda, kind, name, d):
    """Few chains run in 64-thread blocks, many in 256-thread ones."""
    from flowmc_gb300 import targets as TG
    rng = np.random.default_rng(d)
    tgt = {"dual": lambda: TG.DualMoon(d), "rosen": lambda: TG.Rosenbrock(d), "diag": lambda: TG.DiagGaussian(d),
           "mix": lambda: TG.GaussianMixture(rng.normal(size=(3, d)), 0.7)}[name]()
    x = torch.tensor(rng.normal(size=(60000, d)), dtype=torch.float32, device="cuda")
    few, many = _local(tgt, kind, x[:37].contiguous(), 7, 3), _local(tgt, kind, x, 7, 3)
    for a, b in zip(few, many):
        assert torch.equal(a, b[:37])


@pytest.mark.parametrize("a", [20.0, 7.3, 3.0, 1.0000001])
def test_rosenbrock_divisors(cuda, a):
    """Exact quotients by a constant: significands that are even and odd."""
    from flowmc_gb300 import targets as TG
    a = float(np.float32(a))
    tgt = TG.Rosenbrock(10, a=a)
    rng = np.random.default_rng(2)
    C, S = 40, 9
    x0 = rng.normal(size=(C, 10)).astype(np.float32)
    z = rng.normal(size=(C, S, 10)).astype(np.float32)
    u = rng.uniform(1e-6, 1, size=(C, S)).astype(np.float32)
    up = lambda v: torch.tensor(v, device="cuda")
    pos, lp, acc = (v.cpu().numpy() for v in _local(tgt, "mala", up(x0), S, 2, up(z), up(u)))
    op, ol, oa, _ = K.take_serial_steps("mala", tgt.describe(), x0.astype(np.float64), S, z, u, step_size=0.05,
                                        thinning=2)
    ok = (acc == oa).all(1)
    assert ok.mean() >= 0.9
    np.testing.assert_allclose(pos[ok], op[ok], rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(lp[ok], ol[ok], rtol=1e-4, atol=1e-3)


def test_batched_packed_positions(cuda):
    """Positions packed by one launch (float32 rows of any stride, more
    targets than one launch's table holds) and by the general copies (other
    strides and types, broadcast rows): the same chains, bit for bit."""
    from flowmc_gb300 import targets as TG
    from flowmc_gb300.batched import BatchedDenseLocalSteps
    dims = [1, 2, 7, 8, 33, 255, 256] * 10
    chains = [1 + 9 * (i % 5) for i in range(len(dims))]
    ts = [TG.DenseGaussian(np.eye(d) * (1 + 0.1 * i)) for i, d in enumerate(dims)]
    b = BatchedDenseLocalSteps(ts, chains, [0.1] * len(dims))
    g = torch.Generator(device="cuda").manual_seed(4)
    xs = [torch.randn(c, d, device="cuda", generator=g) for c, d in zip(chains, dims)]
    ref = b.pack(xs)
    got = b._packed_rows(xs, xs[0].device)
    strided = [torch.nn.functional.pad(x, (0, 3))[:, :x.shape[1]] for x in xs]
    for t, (x, d) in enumerate(zip(xs, dims)):
        rows = slice(b.offsets[t], b.offsets[t + 1])
        assert torch.equal(got[rows, :d], x) and torch.equal(ref[rows, :d], x)
    runs = [b.run(v, 2, seed=5) for v in (xs, strided, [x.double() for x in xs], [x.t().contiguous().t() for x in xs])]
    for outs, last, lp in runs[1:]:
        for t in range(len(dims)):
            assert all(torch.equal(p, q) for p, q in zip(outs[t], runs[0][0][t]))
            assert torch.equal(last[t], runs[0][1][t]) and torch.equal(lp[t], runs[0][2][t])
