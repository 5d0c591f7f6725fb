"""The work that a user of flowmc_gb300 has it do, as timed cases.

Families (case["family"]):
  local    TakeSerialSteps: a phase of MALA, HMC or random-walk steps over all chains
  global   TakeGroupSteps with NFProposal: flow proposals, their densities and the accept scan
  batched  BatchedDenseLocalSteps: many dense-Gaussian targets of uneven dimension in one call
  flow     MaskedCouplingRQSpline log_prob / inverse / sample over rows
  train    one optimiser step of MaskedCouplingRQSpline: loss, gradient, clipped AdamW
  realnvp  RealNVP log_prob, or its loss and gradient

Sizes are those of the sampler's reference workloads: the 5-D dual moon (20
chains, 4 x [32, 32] flow, float32), the 48 dense Gaussians, the 32-D mixture
flow (8 x [128, 128], 10 bins), the 64-D mixture bundle (4096 chains, 8 x
[256, 256], bf16) and the 128-D Rosenbrock bundle (16,384 chains, 12 x
[512, 512], bf16). ``draw`` spreads over the ranges between them.

In-kernel random numbers and accept decisions have no plain float64
counterpart, so ``exact`` covers the flow, train and realnvp families.
"""
from __future__ import annotations

import math

import numpy as np
import torch

BINS = (4, 5, 6, 8, 10, 12)


def listed():
    return [
        # the smallest calls: the dual-moon example's local phase, global phase and training step
        dict(name="local_dualmoon5", family="local", kernel="mala", target="dualmoon", d=5, chains=20, steps=30,
             thin=1, leapfrog=0, comps=0, step=0.1),
        dict(name="global_dualmoon5_fp32", family="global", target="dualmoon", d=5, chains=20, steps=30, comps=0,
             layers=4, hidden=32, depth=2, bins=8, precision="float32"),
        dict(name="train_dualmoon5_fp32", family="train", d=5, layers=4, hidden=32, depth=2, bins=8, rows=10000,
             precision="float32"),
        # ordinary bundles: local phases of the 64-D mixture and the 128-D Rosenbrock chain
        dict(name="local_mixture64", family="local", kernel="mala", target="mixture", d=64, chains=4096, steps=50,
             thin=1, leapfrog=0, comps=4, step=0.05),
        dict(name="local_rosenbrock128_hmc", family="local", kernel="hmc", target="rosenbrock", d=128, chains=16384,
             steps=40, thin=1, leapfrog=16, comps=0, step=0.01),
        # many posteriors at once: 48 Gaussian targets of 8 to 256 dimensions, 512 to 8192 chains each
        dict(name="batched48_mala", family="batched", kernel="mala", targets=48, d_min=8, d_max=256, c_min=512,
             c_max=8192, steps=10, leapfrog=0, sizes=1),
        dict(name="batched48_hmc", family="batched", kernel="hmc", targets=48, d_min=8, d_max=256, c_min=512,
             c_max=8192, steps=3, leapfrog=10, sizes=1),
        # density evaluation of a fitted float32 flow over a ragged number of rows, and its training step
        dict(name="logprob_mixture32_fp32", family="flow", op="log_prob", d=32, layers=8, hidden=128, depth=2,
             bins=10, rows=100003, precision="float32"),
        dict(name="train_mixture32_fp32", family="train", d=32, layers=8, hidden=128, depth=2, bins=10, rows=16384,
             precision="float32"),
        # the mixture bundle's global phase, and the largest training step
        dict(name="global_mixture64_bf16", family="global", target="mixture", d=64, chains=4096, steps=50, comps=4,
             layers=8, hidden=256, depth=2, bins=8, precision="bf16"),
        dict(name="train_rosenbrock128_bf16", family="train", d=128, layers=12, hidden=512, depth=2, bins=12,
             rows=65536, precision="bf16"),
        # the other flow: loss and gradient of a RealNVP batch
        dict(name="grad_realnvp32", family="realnvp", op="grad", d=32, layers=8, hidden=256, rows=16384),
    ]


# ------------------------------------------------------------------ drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_local(rng):
    target = rng.choice(["dualmoon", "mixture", "rosenbrock", "diag"])
    d = {"dualmoon": lambda: rng.randint(2, 10), "mixture": lambda: _log_int(rng, 8, 128),
         "rosenbrock": lambda: _log_int(rng, 8, 200), "diag": lambda: _log_int(rng, 3, 128)}[target]()
    kernel = rng.choice(["mala", "hmc", "grw"])
    return dict(family="local", kernel=kernel, target=target, d=d, chains=_log_int(rng, 16, 16384),
                steps=rng.randint(10, 50), thin=rng.choice([1, 1, 1, 3, 5]),
                leapfrog=rng.randint(4, 16) if kernel == "hmc" else 0,
                comps=rng.randint(2, 8) if target == "mixture" else 0,
                step=round(rng.uniform(0.01, 0.1), 4))


def _draw_global(rng):
    bf16 = rng.random() < 0.5
    target = rng.choice(["dualmoon", "mixture", "rosenbrock"])
    d = rng.randint(4, 10) if target == "dualmoon" else _log_int(rng, 8, 64 if bf16 else 32)
    return dict(family="global", target=target, d=d, chains=_log_int(rng, 16, 4096 if bf16 else 128),
                steps=rng.randint(10, 50), comps=rng.randint(2, 8) if target == "mixture" else 0,
                layers=rng.randint(2, 8), hidden=rng.choice([64, 128, 256] if bf16 else [16, 24, 32, 64, 128]),
                depth=2, bins=rng.choice([6, 8, 10]), precision="bf16" if bf16 else "float32")


def _draw_batched(rng):
    kernel = rng.choice(["mala", "hmc"])
    return dict(family="batched", kernel=kernel, targets=_log_int(rng, 4, 48), d_min=8,
                d_max=rng.randint(24, 256), c_min=_log_int(rng, 64, 512), c_max=_log_int(rng, 1024, 8192),
                steps=rng.randint(2, 3) if kernel == "hmc" else rng.randint(3, 10),
                leapfrog=rng.randint(3, 10) if kernel == "hmc" else 0, sizes=rng.randint(2, 10 ** 6))


def _draw_flow(rng):
    return dict(family="flow", op=rng.choice(["log_prob", "inverse", "sample"]), d=_log_int(rng, 4, 64),
                layers=rng.randint(2, 8), hidden=rng.choice([16, 24, 32, 50, 64, 100, 128, 256]),
                depth=rng.choice([1, 2, 2, 3]), bins=rng.choice(BINS), rows=_log_int(rng, 1, 100000),
                precision="float32")


def _draw_train(rng):
    bf16 = rng.random() < 0.5
    return dict(family="train", d=_log_int(rng, 4, 128 if bf16 else 40), layers=rng.randint(2, 12 if bf16 else 8),
                hidden=rng.choice([64, 128, 256, 512] if bf16 else [16, 24, 32, 64, 128]), depth=2,
                bins=rng.choice(BINS), rows=_log_int(rng, 500, 65536 if bf16 else 16384),
                precision="bf16" if bf16 else "float32")


def _draw_realnvp(rng):
    return dict(family="realnvp", op=rng.choice(["log_prob", "grad"]), d=_log_int(rng, 4, 64),
                layers=rng.randint(2, 10), hidden=rng.choice([30, 64, 100, 128, 256]),
                rows=_log_int(rng, 100, 16384))


def draw(rng):
    make = rng.choice([_draw_local, _draw_global, _draw_batched, _draw_flow, _draw_train, _draw_realnvp])
    while True:
        case = make(rng)
        same = [c for c in listed() if c["family"] == case["family"] and c.get("precision") == case.get("precision")
                and c.get("kernel") == case.get("kernel")]
        # no dearer than the listed cases of its family, kernel and precision (or, where the family
        # lists none of that kind, than the family's largest)
        same = same or [c for c in listed() if c["family"] == case["family"]]
        w, top = work(case), [work(c) for c in same]
        if w["flops"] <= max(t["flops"] for t in top) and w["bytes"] <= max(t["bytes"] for t in top):
            return case


# ------------------------------------------------------------------ work of one pass
def _eval_flops(target, d, comps):
    """Floating-point operations of one value-and-gradient evaluation of a target."""
    return {"dualmoon": 4 * d + 40, "mixture": comps * (6 * d + 10), "rosenbrock": 15 * d, "diag": 5 * d}[target]


def _flow_flops(case):
    """(GEMM FLOPs per row, spline operations per row) of one pass through a MaskedCouplingRQSpline."""
    d, H, P = case["d"], case["hidden"], 3 * case["bins"] + 1
    gemm = spline = 0
    for layer in range(case["layers"]):
        nc = sum((j + layer) % 2 for j in range(d))
        nt = d - nc
        gemm += 2 * (nc * H + (case["depth"] - 1) * H * H + H * nt * P)
        spline += nt * (6 * P + 40)
    return gemm, spline


def _flow_params(case):
    d, H, P = case["d"], case["hidden"], 3 * case["bins"] + 1
    n = 0
    for layer in range(case["layers"]):
        nc = sum((j + layer) % 2 for j in range(d))
        nt = d - nc
        n += 2 + nc * H + H + (case["depth"] - 1) * (H * H + H) + H * nt * P + nt * P
    return n


def _batched_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    dims = rng.integers(case["d_min"], case["d_max"] + 1, size=case["targets"])
    chains = np.exp(rng.uniform(math.log(case["c_min"]), math.log(case["c_max"]), size=case["targets"])).astype(int)
    return [int(v) for v in dims], [int(v) for v in chains]


def work(case):
    fam = case["family"]
    if fam == "local":
        C, S, d = case["chains"], case["steps"], case["d"]
        rows = C * -(-S // case["thin"])
        evals = C * (S * (case["leapfrog"] + 1 if case["kernel"] == "hmc" else 1) + 1)
        return {"bytes": rows * (4 * d + 8) + C * 8 * d, "flops": evals * (_eval_flops(case["target"], d, case["comps"]) + 4 * d)}
    if fam == "batched":
        dims, chains = _batched_sizes(case)
        evals = case["steps"] * (case["leapfrog"] + 1 if case["kernel"] == "hmc" else 1) + 1
        return {"bytes": sum(c * (case["steps"] * (4 * d + 8) + 8 * d) + 4 * d * d for d, c in zip(dims, chains)),
                "flops": sum(c * evals * (2 * d * d + 4 * d) for d, c in zip(dims, chains))}
    if fam == "realnvp":
        d, H, n = case["d"], case["hidden"], case["rows"]
        fwd = n * case["layers"] * 2 * (4 * H * d)
        params = case["layers"] * (4 * H * d + 2 * H + 2 * d)
        grad = case["op"] == "grad"
        return {"bytes": 4 * (n * d + (1 if grad else n) + params * (2 if grad else 1)), "flops": fwd * (3 if grad else 1)}
    gemm, spline = _flow_flops(case)
    if fam == "global":
        C, S, d = case["chains"], case["steps"], case["d"]
        return {"bytes": C * S * (4 * d + 8) + C * 8 * d + 4 * _flow_params(case),
                "flops": (2 * C * S + C) * (gemm + spline) + C * S * _eval_flops(case["target"], d, case["comps"])}
    n, d = case["rows"], case["d"]
    if fam == "flow":
        out = {"log_prob": 1, "inverse": d + 1, "sample": d}[case["op"]]
        return {"bytes": 4 * (n * (out + (0 if case["op"] == "sample" else d)) + _flow_params(case)),
                "flops": n * (gemm + spline)}
    p = _flow_params(case)   # a training step reads and writes the weights and both moments and writes the gradient
    return {"bytes": 4 * (n * d + 7 * p), "flops": n * 3 * (gemm + spline) + 12 * p}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _mixture_means(d, comps, seed):
    r = np.random.default_rng(seed)
    return 4.0 * np.sqrt(2.0) * np.linalg.qr(r.normal(size=(d, max(comps, 1))))[0].T[:comps] if comps <= d else \
        r.uniform(-4, 4, size=(comps, d))


def _target(case, seed):
    from flowmc_gb300 import targets as T
    d, kind = case["d"], case["target"]
    if kind == "dualmoon":
        return T.DualMoon(d)
    if kind == "rosenbrock":
        return T.Rosenbrock(d)
    if kind == "mixture":
        return T.GaussianMixture(_mixture_means(d, case["comps"], seed), 0.5 * np.ones(d))
    r = np.random.default_rng(seed)
    return T.DiagGaussian(d, mean=r.normal(size=d), inv_var=np.exp(r.uniform(-1, 1, size=d)))


def _start(case, seed, g):
    """Chains inside the target's bulk, as after the first loops."""
    C, d, kind = case["chains"], case["d"], case["target"]
    z = _randn(g, C, d)
    if kind == "dualmoon":
        return 2.0 * z / z.norm(dim=1, keepdim=True) * (1.0 + 0.05 * _randn(g, C, 1))
    if kind == "rosenbrock":
        return 0.3 * z + 0.5
    if kind == "mixture":
        mu = torch.tensor(_mixture_means(d, case["comps"], seed), dtype=torch.float32, device="cuda")
        return mu[torch.randint(0, case["comps"], (C,), generator=g, device="cuda")] + math.sqrt(0.5) * z
    return z


def _flow_data(case, rows, g):
    """Training-like rows: an eight-component mixture with unequal scales."""
    d = case["d"]
    mu = torch.empty(8, d, device="cuda").uniform_(-5, 5, generator=g)
    sd = torch.empty(8, d, device="cuda").uniform_(0.3, 1.0, generator=g)
    k = torch.randint(0, 8, (rows,), generator=g, device="cuda")
    return mu[k] + sd[k] * _randn(g, rows, d)


def _flow_sizes(case, layer):
    d = case["d"]
    nc = sum((j + layer) % 2 for j in range(d))
    ins = [nc] + [case["hidden"]] * case["depth"]
    outs = [case["hidden"]] * case["depth"] + [(d - nc) * (3 * case["bins"] + 1)]
    return list(zip(outs, ins))


def _flow_theta(case, g):
    """A partly trained flow's packed parameters: scale, shift, then W and b of each Linear, per layer."""
    parts = []
    for layer in range(case["layers"]):
        parts.append(0.02 * _randn(g, 2))
        for o, i in _flow_sizes(case, layer):
            parts += [_randn(g, o * i) * (0.7 / math.sqrt(i)), 0.1 * _randn(g, o)]
    return torch.cat(parts)


def _flow_inputs(case, rows, seed):
    g = _gen(seed)
    theta = _flow_theta(case, g)
    x = _flow_data(case, max(rows, 64), g)
    return theta, x.mean(0), x.var(0), x[:rows].contiguous()


def _flow_model(case, theta, mean, var):
    from flowmc_gb300.api import MaskedCouplingRQSpline, PRNGKey
    m = MaskedCouplingRQSpline(case["d"], case["layers"], [case["hidden"]] * case["depth"], case["bins"], PRNGKey(0),
                               precision=case["precision"], device="cuda")
    m.theta.copy_(theta)
    m.aux[: case["d"]] = mean
    m.aux[case["d"]: 2 * case["d"]] = var
    m.sync_bf16()
    return m


def _rnvp_theta(case, g):
    d, H = case["d"], case["hidden"]
    parts = []
    for _ in range(case["layers"]):
        parts += [_randn(g, 2 * H * d) * (0.7 / math.sqrt(d)), 0.1 * _randn(g, 2 * H)]
        for _ in range(2):
            parts += [_randn(g, d * H) * (0.2 / math.sqrt(H)), 0.02 * _randn(g, d)]
    return torch.cat(parts)


def _adam_state(n, g):
    """Moments of an optimiser some hundred steps in."""
    return 1e-4 * _randn(g, n), 1e-7 * (0.5 + torch.rand(n, generator=g, device="cuda")), 200


def _stepper_state(case, seed):
    """Buffers, target and strategy state of one sampling phase."""
    from flowmc_gb300.api import Buffer, LogPDF, State
    C, d = case["chains"], case["d"]
    rows = -(-case["steps"] // case.get("thin", 1))
    bufs = [Buffer("positions", (C, rows, d), 1), Buffer("log_prob", (C, rows), 1), Buffer("accepts", (C, rows), 1)]
    res = {b.name: b for b in bufs}
    res["logpdf"] = LogPDF(_target(case, seed), n_dims=d)
    res["state"] = State({"p": "positions", "l": "log_prob", "a": "accepts"})
    return res


def prepare(case, seed):
    from flowmc_gb300 import api
    fam = case["family"]
    if fam in ("local", "global"):
        g = _gen(seed)
        res = _stepper_state(case, seed)
        x0 = _start(case, seed, g)
        if fam == "local":
            res["kernel"] = {"mala": lambda: api.MALA(case["step"]), "grw": lambda: api.GaussianRandomWalk(case["step"]),
                             "hmc": lambda: api.HMC(1, case["step"], case["leapfrog"])}[case["kernel"]]()
            stepper = api.TakeSerialSteps("logpdf", "kernel", "state", ["p", "l", "a"], case["steps"],
                                          thinning=case["thin"])
        else:
            x = x0 if x0.shape[0] >= 64 else x0.repeat(4, 1)
            # a flow fitted well enough to be accepted now and then: weights kept small about the data's moments
            theta = 0.3 * _flow_theta(case, g)
            res["kernel"] = api.NFProposal(_flow_model(case, theta, x.mean(0), x.var(0) + 1e-3))
            stepper = api.TakeGroupSteps("logpdf", "kernel", "state", ["p", "l", "a"], case["steps"])
        return dict(family=fam, res=res, x0=x0, stepper=stepper, key=api.PRNGKey(seed))
    if fam == "batched":
        from flowmc_gb300.batched import BatchedDenseLocalSteps
        dims, chains = _batched_sizes(case)
        g, tg, steps, xs = _gen(seed), [], [], []
        for d, c in zip(dims, chains):
            lam = torch.exp(torch.empty(d, device="cuda").uniform_(math.log(1e-2), math.log(10.0), generator=g)).double()
            q = torch.linalg.qr(_randn(g, d, d).double())[0]
            tg.append(api.targets.DenseGaussian(((q / lam) @ q.T).cpu().numpy()))
            s = float(lam.min()) ** 0.5
            steps.append(0.2 * s if case["kernel"] == "hmc" else 0.5 * s * d ** (-1 / 3))
            xs.append(((q * lam.sqrt()) @ _randn(g, d, c).double()).T.float().contiguous())
        runner = BatchedDenseLocalSteps(tg, chains, steps, kind=case["kernel"], n_leapfrog=case["leapfrog"] or 10)
        S = case["steps"]
        # one block of memory per kind of row; each target's buffer is an aligned slice of it
        cut = lambda sizes: [sum(sizes[:i]) for i in range(len(sizes) + 1)]
        po = cut([-(-c * S * d // 128) * 128 for d, c in zip(dims, chains)])
        so = cut([-(-c * S // 128) * 128 for c in chains])
        pos, lp, acc = (torch.zeros(n, device="cuda") for n in (po[-1], so[-1], so[-1]))
        outs = [(pos[po[i]:po[i] + c * S * d].view(c, S, d), lp[so[i]:so[i] + c * S].view(c, S),
                 acc[so[i]:so[i] + c * S].view(c, S)) for i, (d, c) in enumerate(zip(dims, chains))]
        return dict(family=fam, runner=runner, xs=xs, steps=S, outs=outs, flat=(pos, lp, acc), seed=seed)
    if fam == "realnvp":
        g = _gen(seed)
        theta, x = _rnvp_theta(case, g), _flow_data(case, case["rows"], g)
        m = api.RealNVP(case["d"], case["layers"], case["hidden"], api.PRNGKey(0), device="cuda")
        m.theta.copy_(theta)
        m.aux[: case["d"]] = 0.0
        m.aux[case["d"]: 2 * case["d"]] = 10.0
        return dict(family=fam, op=case["op"], model=m, x=x)
    theta, mean, var, x = _flow_inputs(case, case["rows"], seed)
    model = _flow_model(case, theta, mean, var)
    if fam == "flow":
        if case["op"] == "inverse":
            x = (x - mean) / var.sqrt()
        return dict(family=fam, op=case["op"], model=model, x=x, key=api.PRNGKey(seed))
    opt = api.Optimizer(model, learning_rate=1e-3)
    m, v, count = _adam_state(theta.numel(), _gen(seed + 1))
    opt.optim_state.m.copy_(m)
    opt.optim_state.v.copy_(v)
    opt.optim_state.count.fill_(count)
    return dict(family=fam, model=model, x=x, opt=opt, loss=torch.empty((), device="cuda"),
                grad=torch.empty_like(model.theta))


# ------------------------------------------------------------------ one pass
def run(state):
    fam = state["family"]
    if fam in ("local", "global"):
        st, res = state["stepper"], state["res"]
        st.set_current_position(0)
        _, _, last = st(state["key"], res, state["x0"], {})
        return {"positions": res["positions"].data, "log_prob": res["log_prob"].data, "accepts": res["accepts"].data,
                "last": last}
    if fam == "batched":
        state["runner"].run(state["xs"], state["steps"], seed=state["seed"], outputs=state["outs"])
        return state["flat"]
    m, x = state["model"], state["x"]
    if fam == "realnvp":
        return m.log_prob(x) if state["op"] == "log_prob" else m.loss_and_grad(x)
    if fam == "flow":
        if state["op"] == "sample":
            return m.sample(state["key"], x.shape[0])
        return m.log_prob(x) if state["op"] == "log_prob" else m.inverse(x)
    loss, grad = m.loss_and_grad(x, state["loss"], state["grad"])
    state["opt"].apply(m, grad, state["opt"].optim_state)
    return {"loss": loss, "grad": grad, "theta": m.theta}


# ------------------------------------------------------------------ float64
def _spline64(x, raw, K, inverse):
    """Rational-quadratic spline on [-10, 10] with linear tails: (output, log-derivative), plain float64 torch."""
    lo, hi, min_bin, min_slope = -10.0, 10.0, 1e-4, 1e-4
    size = lambda r: torch.softmax(r, -1) * ((hi - lo) - K * min_bin) + min_bin
    edge = lambda w: torch.cat([torch.full_like(w[..., :1], lo), lo + torch.cumsum(w[..., :-1], -1),
                                torch.full_like(w[..., :1], hi)], -1)
    xp, yp = edge(size(raw[..., :K])), edge(size(raw[..., K:2 * K]))
    sl = torch.nn.functional.softplus(raw[..., 2 * K:] + math.log(math.exp(1.0 - min_slope) - 1.0)) + min_slope
    at = yp if inverse else xp
    k = (torch.searchsorted(at.detach().contiguous(), x.detach()[..., None].contiguous(), right=True) - 1).clamp(0, K - 1)
    pick = lambda a, kk: torch.gather(a, -1, kk)[..., 0]
    x0, x1, y0, y1, d0, d1 = (pick(a, k + o) for a, o in ((xp, 0), (xp, 1), (yp, 0), (yp, 1), (sl, 0), (sl, 1)))
    w, h = x1 - x0, y1 - y0
    s = h / w
    if inverse:
        t = ((x - y0) / h).clamp(0, 1)
        b = d0 - (d1 + d0 - 2 * s) * t
        a, c = s - b, -s * t
        disc = (b * b - 4 * a * c).clamp_min(0).sqrt()
        z = torch.where(b >= 0, 2 * c / (-b - disc), (-b + disc) / (2 * a)).clamp(0, 1)
    else:
        z = ((x - x0) / w).clamp(0, 1)
    q = z * (1 - z)
    den = s + (d1 + d0 - 2 * s) * q
    ld = 2 * torch.log(s) + torch.log(d1 * z * z + 2 * s * q + d0 * (1 - z) ** 2) - 2 * torch.log(den)
    out = w * z + x0 if inverse else y0 + h * (s * z * z + d0 * q) / den
    first, last = sl[..., 0], sl[..., -1]
    below, above = x <= at[..., 0], x >= at[..., -1]
    if inverse:
        out = torch.where(below, (x - lo) / first + lo, torch.where(above, (x - hi) / last + hi, out))
    else:
        out = torch.where(below, (x - lo) * first + lo, torch.where(above, (x - hi) * last + hi, out))
    ld = torch.where(below, torch.log(first), torch.where(above, torch.log(last), ld))
    return out, -ld if inverse else ld


def _flow64(case, theta, x, inverse=False):
    """The coupling layers in float64: (output, log-determinant)."""
    d, K = case["d"], case["bins"]
    P = 3 * K + 1
    off, layers = 0, []
    for layer in range(case["layers"]):
        scale, shift = theta[off], theta[off + 1]
        off += 2
        lin = []
        for o, i in _flow_sizes(case, layer):
            lin.append((theta[off:off + o * i].view(o, i), theta[off + o * i:off + o * i + o]))
            off += o * i + o
        layers.append((layer, scale, shift, lin))
    ld = torch.zeros(x.shape[0], dtype=x.dtype, device=x.device)
    for layer, scale, shift, lin in reversed(layers) if inverse else layers:
        x = x * torch.exp(-scale) - shift if inverse else (x + shift) * torch.exp(scale)
        ld = ld + (-d * scale if inverse else d * scale)
        cond = [j for j in range(d) if (j + layer) % 2]
        move = [j for j in range(d) if not (j + layer) % 2]
        a = x[:, cond]
        for n, (W, b) in enumerate(lin):
            a = a @ W.T + b
            if n < len(lin) - 1:
                a = torch.tanh(a)
        y, l = _spline64(x[:, move], a.view(x.shape[0], len(move), P), K, inverse)
        x = torch.zeros_like(x).index_copy(1, torch.tensor(cond, device=x.device), x[:, cond]).index_copy(
            1, torch.tensor(move, device=x.device), y)
        ld = ld + l.sum(-1)
    return x, ld


def _flow_logprob64(case, theta, mean, var, x):
    y, ld = _flow64(case, theta, (x - mean) / var.sqrt())
    return ld - 0.5 * (y * y).sum(-1) - 0.5 * case["d"] * math.log(2 * math.pi)


def _rnvp_logprob64(case, theta, x):
    d, H = case["d"], case["hidden"]
    y, ld, off = x / math.sqrt(10.0), 0.0, 0

    def take(*shape):
        nonlocal off
        n = math.prod(shape)
        off += n
        return theta[off - n:off].view(*shape)

    for layer in range(case["layers"]):
        W1, b1 = take(2 * H, d), take(2 * H)
        W2s, b2s, W2t, b2t = take(d, H), take(d), take(d, H), take(d)
        m = torch.zeros(d, dtype=x.dtype, device=x.device)
        m[: d // 2] = 1.0
        m = m if layer % 2 == 0 else 1 - m
        h = torch.relu((y * m) @ W1.T + b1)
        s = torch.tanh(h[:, :H] @ W2s.T + b2s)
        t = h[:, H:] @ W2t.T + b2t
        y = (1 - m) * ((y + t) * torch.exp(s)) + m * y
        ld = ld + ((1 - m) * s).sum(-1)
    return ld - 0.5 * (y * y).sum(-1) - 0.5 * d * math.log(2 * math.pi)


def _loss_grad64(logprob, theta, x, chunk):
    """Mean negative log-density and its gradient, accumulated over row chunks."""
    theta = theta.double().requires_grad_(True)
    loss, grad = 0.0, torch.zeros_like(theta)
    for r in range(0, x.shape[0], chunk):
        part = -logprob(theta, x[r:r + chunk].double()).sum() / x.shape[0]
        grad += torch.autograd.grad(part, theta)[0]
        loss = loss + part.detach()
    return loss, grad


def exact(case, seed):
    fam = case["family"]
    if work(case)["flops"] > 3e12:   # float64 runs at about 1 TFLOP/s, and autograd keeps every spline intermediate
        return None
    if fam == "realnvp":
        g = _gen(seed)
        theta, x = _rnvp_theta(case, g), _flow_data(case, case["rows"], g)
        if case["op"] == "log_prob":
            return _rnvp_logprob64(case, theta.double(), x.double())
        return _loss_grad64(lambda th, v: _rnvp_logprob64(case, th, v), theta, x, 16384)
    if fam == "flow":
        if case["op"] == "sample":   # the base normals are drawn inside the call
            return None
        theta, mean, var, x = _flow_inputs(case, case["rows"], seed)
        out = []
        for r in range(0, x.shape[0], 16384):
            v = x[r:r + 16384]
            if case["op"] == "log_prob":
                out.append((_flow_logprob64(case, theta.double(), mean.double(), var.double(), v.double()),))
            else:
                out.append(_flow64(case, theta.double(), ((v - mean) / var.sqrt()).double(), inverse=True))
        out = [torch.cat(o) for o in zip(*out)]
        return out[0] if case["op"] == "log_prob" else tuple(out)
    if fam == "train":
        theta, mean, var, x = _flow_inputs(case, case["rows"], seed)
        m64, v64 = mean.double(), var.double()
        loss, grad = _loss_grad64(lambda th, v: _flow_logprob64(case, th, m64, v64, v), theta, x, 4096)
        # clip to a global norm of 1, then AdamW (b1 0.9, b2 0.999, eps 1e-8, decay 1e-4, rate 1e-3)
        m, v, count = _adam_state(theta.numel(), _gen(seed + 1))
        g = grad / max(1.0, float(grad.norm()))
        m, v, t = 0.9 * m.double() + 0.1 * g, 0.999 * v.double() + 0.001 * g * g, count + 1
        step = (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8) + 1e-4 * theta.double()
        return {"loss": loss, "grad": grad, "theta": theta.double() - 1e-3 * step}
    return None   # sampling phases: noise drawn in the kernels, accept decisions
