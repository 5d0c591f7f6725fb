"""Tile edges of the batched dense-Gaussian kernel: dimensions at and beside
the 32-coordinate block, the 8- and 16-row stages of P and the tile's widest
shape, chain counts that leave a row block part empty, non-zero means and
thinning, against the oracle; and the tile height, which follows the total
work, never changes a chain's bits."""
import numpy as np
import pytest
import torch

from oracle import kernels as K

pytestmark = pytest.mark.gpu


def make(dims, seed):
    from flowmc_gb300 import targets as TG
    rng = np.random.default_rng(seed)
    ts, steps = [], []
    for d in dims:
        Q = np.linalg.qr(rng.normal(size=(d, d)))[0]
        lam = np.exp(rng.uniform(np.log(0.1), np.log(2.0), size=d))
        ts.append(TG.DenseGaussian((Q / lam) @ Q.T, mean=rng.normal(size=d), const=0.25, device="cuda"))
        steps.append(0.3 * float(np.sqrt(lam.min())) * d ** (-1 / 6))
    return ts, steps


@pytest.mark.parametrize("kind,nlf", [("mala", 0), ("hmc", 3)])
def test_tile_edges_match_oracle(cuda, kind, nlf):
    from flowmc_gb300.batched import BatchedDenseLocalSteps
    dims = [1, 8, 9, 31, 32, 33, 96, 97, 224, 225, 255]
    chains = [33, 1, 400, 65, 64, 32, 31, 100, 5, 40, 33]
    ts, steps = make(dims, 4)
    S, thin = 5, 2
    rng = np.random.default_rng(6)
    xs = [rng.normal(size=(c, d)).astype(np.float32) for c, d in zip(chains, dims)]
    nz = [rng.normal(size=(c, S, d)).astype(np.float32) for c, d in zip(chains, dims)]
    un = [rng.uniform(1e-6, 1, size=(c, S)).astype(np.float32) for c in chains]
    up = lambda v: [torch.tensor(a, device="cuda") for a in v]
    b = BatchedDenseLocalSteps(ts, chains, steps, kind=kind, n_leapfrog=nlf)
    outs, last, lp_last = b.run(up(xs), S, thinning=thin, noise=up(nz), uniform=up(un))
    same = total = 0
    for t, d in enumerate(dims):
        pos, lp, acc = (o.cpu().numpy() for o in outs[t])
        opos, olp, oacc, olast = K.take_serial_steps(kind, ts[t].describe(), xs[t].astype(np.float64), S,
                                                     nz[t].astype(np.float64), un[t].astype(np.float64),
                                                     step_size=steps[t], n_leapfrog=nlf, M=np.eye(d), thinning=thin)
        ok = (acc == oacc).all(1)           # chains without a tie flip
        same, total = same + int(ok.sum()), total + len(ok)
        np.testing.assert_allclose(pos[ok], opos[ok], rtol=1e-4, atol=1e-4)
        np.testing.assert_allclose(lp[ok], olp[ok], rtol=1e-4, atol=1e-3)
        np.testing.assert_array_equal(last[t].cpu().numpy(), pos[:, -1])
        np.testing.assert_array_equal(lp_last[t].cpu().numpy(), lp[:, -1])
    assert same >= 0.95 * total


@pytest.mark.parametrize("kind", ["mala", "hmc"])
@pytest.mark.parametrize("d", [20, 50, 130])
def test_tile_height_does_not_change_a_chain(cuda, kind, d):
    from flowmc_gb300.batched import BatchedDenseLocalSteps
    ts, steps = make([d, 40], 9)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    xs = [torch.randn(c, dd, device="cuda", generator=g) for c, dd in ((1000, d), (60000, 40))]
    one = BatchedDenseLocalSteps(ts[:1], [1000], steps[:1], kind=kind, n_leapfrog=2).run(xs[:1], 3, seed=8)
    two = BatchedDenseLocalSteps(ts, [1000, 60000], steps, kind=kind, n_leapfrog=2).run(xs, 3, seed=8)
    for a, b in zip(one[0][0], two[0][0]):
        assert torch.equal(a, b)
