"""Performance cases: the calls a user of this framework makes, over the sizes they make them at.

A case is a dict of plain values; `prepare` builds what the caller's program holds before the call (an
engine, generation tables, rows, network weights, page-locked result buffers), `run` is one pass through
the public entry points and returns its whole outputs, `work` says what the pass cannot do without and
`exact` what it returns in 64-bit arithmetic (where that is defined without simulating).

Kinds:
    sim        one simulation: equilibrium start, generations with compactions (and time samples), final
               state to page-locked host arrays, spectrum of each population
    spectra    mean spectra of many small replicates (the batched engine through simulate_spectra)
    sfs        projected spectrum of one frequency row, on the device or through host arrays
    hist       population histogram of one host row
    joint      joint spectrum of two or three populations' rows
    forward    surrogate network inference on a device batch
    gradients  loss and gradients of one batch
    train      minibatch training steps, then the weights
    query      surrogate queries, host parameters in and host spectra out
"""
from __future__ import annotations

import math

import numpy as np
import torch

from parallelpopgen_b200 import ConstantModel, Engine, constant_generations
from parallelpopgen_b200 import surrogate as sg

LAYERS = ((512, 6), (512, 512), (512, 512), (512, 512), (99, 512))


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def sim(name, N, L, gens, n, mu=1e-9, gamma=0.0, h=0.5, F=0.0, P=1, m=0.0, compact=25, samples=0):
    case = {"kind": "sim", "N": N, "L": float(L), "mu": mu, "gens": gens, "n": n, "gamma": gamma, "h": h, "F": F,
            "P": P, "m": m, "compact": compact, "samples": samples}
    return {"name": name, **case} if name else case


def listed():
    return [
        # a quick look at a model: a few hundred mutations, 200 generations -- launch latency only
        sim("sim_small", N=2_000, mu=1e-8, L=1e6, gens=200, n=50),
        # the usual single-population run: N = 1e4, a 20 Mb region, 1,000 generations, sample of 100
        sim("sim_medium", N=10_000, L=2e7, gens=1_000, n=100),
        # the benchmark's two halves (N = 2e5, 250 Mb each; neutral, then purifying selection), a stretch of
        # their 10,000 generations, with the spectrum of 1,000
        sim("sim_large_neutral", N=200_000, L=2.5e8, gens=500, n=1_000),
        sim("sim_large_selected", N=200_000, L=2.5e8, gens=500, n=1_000, gamma=-10.0),
        # three populations exchanging migrants, inbreeding and dominance, a time sample every 100
        # generations (each preserves its survivors, so the state keeps growing)
        sim("sim_three_populations", N=50_000, L=1e8, gens=400, n=200, P=3, m=1e-4, gamma=-5.0, h=0.3, F=0.1,
            compact=35, samples=4),
        # training data for the surrogate: 32 parameter draws x 16 replicates in one batch
        {"name": "spectra_512", "kind": "spectra", "draws": 32, "reps": 16},
        # the spectrum of 1,000 of a large state already on the device
        {"name": "sfs_large", "kind": "sfs", "N": 131_072, "M": 2_700_000, "n": 1_000, "where": "device"},
        # joint spectra of simulated populations: the sample sizes of a two- and a three-population study
        {"name": "joint_two", "kind": "joint", "M": 200_000, "na": 100, "nb": 80, "nc": 0},
        {"name": "joint_three", "kind": "joint", "M": 100_000, "na": 20, "nb": 16, "nc": 12},
        # a sweep of the parameter space through the network: the benchmark's 32,768 queries on the device
        {"name": "forward_32768", "kind": "forward", "batch": 32_768},
        # training the network: 50 minibatches of 1,024
        {"name": "train_1024", "kind": "train", "rows": 16_384, "batch": 1_024, "steps": 50},
        # queries of a host program (an optimiser, a likelihood surface)
        {"name": "query_4096", "kind": "query", "count": 4_096},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["sim"] * 5 + ["spectra", "sfs", "sfs", "hist", "joint", "joint", "forward", "gradients",
                                     "train", "query"])
    if kind == "sim":
        P = rng.choice([1, 1, 1, 1, 2, 3, 4, 6])
        N = int(_log(rng, 500, 2e5))
        mu = 1e-9 if N >= 5_000 else 1e-8
        theta = _log(rng, 20.0, 2e5 / P ** 2)               # 2 mu (2N) L
        slots = P * theta * (math.log(2 * N) + 0.6)
        gens = int(min(_log(rng, 50, 1_000), max(50.0, 1.2e9 / (P * slots))))
        return sim(None, N=N, mu=mu, L=max(1e4, round(theta / (4 * mu * N))), gens=gens,
                   n=int(_log(rng, 20, min(1_000, N))), gamma=rng.choice([0.0, round(rng.uniform(-50, 10), 3)]),
                   h=round(rng.uniform(0, 1), 3), F=rng.choice([0.0, round(rng.uniform(0, 0.5), 3)]), P=P,
                   m=0.0 if P == 1 else round(_log(rng, 1e-5, 1e-2), 7), compact=rng.choice([25, 35, rng.randint(5, 40)]),
                   samples=rng.choice([0, 0, 1, 3]))
    if kind == "spectra":
        return {"kind": "spectra", "draws": rng.randint(2, 32), "reps": rng.randint(1, 16)}
    if kind == "sfs":
        # power-of-two sizes: their grid is exact in every division; other rows are projected one by one
        N = 2 ** rng.randint(10, 17) if rng.random() < 0.6 else int(_log(rng, 1e3, 2e5))
        M = int(_log(rng, 1e3, 2.7e6))
        n = int(_log(rng, 10, min(1_023, N)))
        if N & (N - 1):
            M = min(M, int(3e8 / n))
        return {"kind": "sfs", "N": N, "M": M, "n": n, "where": rng.choice(["device", "host"])}
    if kind == "hist":
        return {"kind": "hist", "N": int(_log(rng, 500, 2e5)), "M": int(_log(rng, 1e3, 2.7e6))}
    if kind == "joint":
        if rng.random() < 0.5:
            na, nb, nc = int(_log(rng, 5, 200)), int(_log(rng, 5, 200)), 0
        else:
            na, nb, nc = (int(_log(rng, 4, 40)) for _ in range(3))
        bins = (na + 1) * (nb + 1) * (nc + 1)
        return {"kind": "joint", "M": int(min(_log(rng, 1e3, 2e5), 3e9 / bins)), "na": na, "nb": nb, "nc": nc}
    if kind == "forward":
        return {"kind": "forward", "batch": 128 * int(_log(rng, 1, 256))}
    if kind == "gradients":
        return {"kind": "gradients", "batch": 128 * int(_log(rng, 1, 64))}
    if kind == "train":
        return {"kind": "train", "rows": 16_384, "batch": 128 * rng.randint(1, 32), "steps": rng.randint(5, 50)}
    return {"kind": "query", "count": int(_log(rng, 1, 16_384))}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _generator(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _counts(seed, M, Nc):
    """Allele counts with the neutral spectrum's density 1/j over 1 .. Nc - 1."""
    u = torch.rand(M, generator=_generator(seed), device="cuda", dtype=torch.float64)
    return torch.clamp(torch.floor(torch.exp(u * math.log(Nc))), 1, Nc - 1).to(torch.int64)


def _row(case, seed):
    """One population's frequency row, with one mutation in a hundred lost or fixed."""
    Nc = 2 * case["N"]
    j = _counts(seed, case["M"], Nc)
    u = torch.rand(case["M"], generator=_generator(seed + 1), device="cuda")
    j = torch.where(u < 0.008, torch.zeros_like(j), torch.where(u < 0.01, torch.full_like(j, Nc), j))
    return j.float() / float(Nc)


def _joint_rows(case, seed):
    """Rows of the same mutations in each population: half private to one of them, the rest shared with
    correlated frequencies, a few fixed in one."""
    P, M, Nc = (3 if case["nc"] else 2), case["M"], 20_000
    j = _counts(seed, M, Nc).double()
    g = _generator(seed + 1)
    rows = []
    private = torch.rand(M, generator=g, device="cuda") < 0.5
    owner = torch.randint(0, P, (M,), generator=g, device="cuda")
    for p in range(P):
        wobble = torch.exp(0.5 * torch.randn(M, generator=g, device="cuda", dtype=torch.float64))
        jp = torch.clamp(torch.round(j * wobble), 0, Nc)
        jp = torch.where(private & (owner != p), torch.zeros_like(jp), jp)
        rows.append((jp.float() / float(Nc)).contiguous())
    return rows


def _weights(seed):
    """He-uniform weights (a smaller output layer), small biases, flat in layer order."""
    g = _generator(seed, "cpu")
    parts = []
    for i, (r, c) in enumerate(LAYERS):
        bound = math.sqrt((6.0 if i < 4 else 1.0) / c)
        parts.append((torch.rand(r * c, generator=g) * 2 - 1) * bound)
        parts.append(torch.randn(r, generator=g) * 0.05)
    return torch.cat(parts)


def _xy(seed, rows):
    """Network inputs over the scaled box and smooth standardised targets of them."""
    g = _generator(seed + 1)
    x = torch.rand((rows, 6), generator=g, device="cuda") * 2 - 1
    f = torch.arange(1, 100, device="cuda") / 100.0
    t = torch.sin(2 * x[:, :1] + 3 * f) * x[:, 1:2] + 0.5 * x[:, 2:3] * f + 0.1 * torch.cos(4 * x[:, 3:4] * f)
    return x.contiguous(), t.float().contiguous()


def _parameters(seed, count):
    """Model parameters over the surrogate's support box: (log N, gamma, h, F, r, T)."""
    low = np.array([math.log(1e3), -100.0, 0.0, 0.0, -0.001, 0.05])
    high = np.array([math.log(1e4), 10.0, 1.0, 0.5, 0.01, 1.0])
    return low + (high - low) * np.random.default_rng(seed).uniform(size=(count, 6))


def _scale(seed):
    """Mean and spread per bin of standardised log spectra."""
    k = np.arange(1, 100)
    rng = np.random.default_rng(seed)
    return -np.log(k) - 1.7 + 0.05 * rng.normal(size=99), 0.3 + 0.3 * rng.uniform(size=99)


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sim":
        N, P, G = case["N"], case["P"], case["gens"]
        s = ConstantModel.s_from_gamma(case["gamma"], N, case["F"]) if case["gamma"] else 0.0
        model = ConstantModel(N=N, F=case["F"], h=case["h"], s=s, mu=case["mu"], P=P, m=case["m"])
        k = case["samples"]
        ends = [G * (i + 1) // k for i in range(k)] if k else []
        segments, last, next_compact = [], 0, case["compact"]
        for end in ends or [G]:
            gens = constant_generations(model, last + 1, end - last, case["compact"], next_compact=next_compact)
            if k:   # a time sample: compaction that preserves its survivors
                gens["preserve"][-1] = 1
            segments.append(gens)
            last, next_compact = end, end + case["compact"]
        theta = 4.0 * case["mu"] * N * case["L"]
        room = int(P * theta * (math.log(2 * N) + 0.6) * (1.5 + k) * (2 if case["gamma"] > 0 else 1)) + 20_000
        bufs = [(_pinned(P * room, torch.float32), _pinned((room, 4), torch.int32)) for _ in segments]
        sfs = _pinned((P, case["n"]), torch.float32)
        return {"case": case, "engine": Engine(), "model": model, "pops": model.mse_pops(), "segments": segments,
                "bufs": [(f.numpy(), i.numpy()) for f, i in bufs], "tensors": bufs, "sfs": sfs,
                "d_sfs": torch.empty((P, case["n"]), dtype=torch.float32, device="cuda"),
                "seed1": 0xBEEF + 2 * seed, "seed2": 0xDECAF - 2 * seed}
    if kind == "spectra":
        return {"case": case, "engine": Engine(), "params": _parameters(seed, case["draws"]), "seed": (seed % 1000) << 20}
    if kind in ("sfs", "hist"):
        row = _row(case, seed)
        host = kind == "hist" or case["where"] == "host"
        st = {"case": case, "engine": Engine(), "row": row.cpu().numpy() if host else row, "Nc": 2 * case["N"],
              "L": float(20 * case["M"])}
        if not host:
            st["out"] = torch.empty(case["n"], dtype=torch.float32, device="cuda")
        return st
    if kind == "joint":
        rows = _joint_rows(case, seed)
        st = {"case": case, "engine": Engine(), "L": float(20 * case["M"])}
        if case["nc"]:
            return {**st, "rows": [r.cpu().numpy() for r in rows]}
        return {**st, "rows": rows, "out": torch.empty((case["na"] + 1, case["nb"] + 1), dtype=torch.float32, device="cuda")}
    if kind in ("forward", "gradients"):
        mlp = sg.Mlp(capacity=case["batch"])
        mlp.set_params(_weights(seed).numpy())
        x, t = _xy(seed, case["batch"])
        return {"case": case, "mlp": mlp, "x": x, "t": t}
    if kind == "train":
        mlp = sg.Mlp(capacity=max(512, case["batch"]), lr=1e-3)
        mlp.set_params(_weights(seed).numpy())
        x, t = _xy(seed, case["rows"])
        return {"case": case, "mlp": mlp, "x": x, "t": t, "seed": seed}
    mlp = sg.Mlp(capacity=32_768)
    mlp.set_params(_weights(seed).numpy())
    mean, std = _scale(seed)
    return {"case": case, "surrogate": sg.Surrogate(mlp, Engine(), scale=sg.TargetScale(mean, std)),
            "params": _parameters(seed, case["count"])}


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sim":
        return _run_sim(state)
    if kind == "spectra":
        mean, var = sg.simulate_spectra(state["engine"], state["params"], case["reps"], state["seed"], with_variance=True)
        return {"mean": mean, "var": var}
    if kind == "sfs":
        e, row = state["engine"], state["row"]
        if case["where"] == "host":
            return {"sfs": e.site_frequency_spectrum(row, state["Nc"], case["n"], state["L"])}
        e.site_frequency_spectrum_device(row.data_ptr(), row.numel(), state["Nc"], case["n"], state["L"],
                                         state["out"].data_ptr())
        e.synchronize()
        return {"sfs": state["out"]}
    if kind == "hist":
        return {"hist": state["engine"].population_histogram(state["row"], state["Nc"], state["L"])}
    if kind == "joint":
        e, rows = state["engine"], state["rows"]
        if case["nc"]:
            return {"joint": e.joint3_site_frequency_spectrum(*rows, case["na"], case["nb"], case["nc"], state["L"])}
        e.joint_site_frequency_spectrum_device(rows[0].data_ptr(), rows[1].data_ptr(), case["M"], case["na"], case["nb"],
                                               state["L"], state["out"].data_ptr())
        e.synchronize()
        return {"joint": state["out"]}
    if kind == "forward":
        return {"y": state["mlp"].forward(state["x"])}
    if kind == "gradients":
        grads, loss = state["mlp"].gradients(state["x"], state["t"])
        return {"grads": grads, "loss": loss}
    if kind == "train":
        sg.train(state["mlp"], state["x"], state["t"], steps=case["steps"], batch=case["batch"], seed=state["seed"],
                 log_every=0)
        return {"weights": state["mlp"].get_params()}
    p, routed = state["surrogate"].query(state["params"])
    return {"p": p, "routed": routed}


def _run_sim(state):
    case, e = state["case"], state["engine"]
    P, Nc = case["P"], state["model"].Nchrom_e
    e.begin_mse(state["pops"], seed1=state["seed1"], seed2=state["seed2"], num_sites=case["L"],
                compact_interval=case["compact"])
    out, flying = {}, None

    def rows(k, M):   # the caller's arrays: rows packed [P][M], IDs [M][4], zeros behind them
        out["M%d" % k], (out["freq%d" % k], out["ids%d" % k]) = M, state["tensors"][k]

    last = len(state["segments"]) - 1
    for k, gens in enumerate(state["segments"]):
        e.run(gens)
        if flying is not None:
            rows(flying, e.sample_wait())
            flying = None
        if k < last:
            e.sample_begin(*state["bufs"][k])
            flying = k
    d_freq, stride, M = e.device_state()
    for p in range(P):
        e.site_frequency_spectrum_device(d_freq + 4 * p * stride, M, Nc, case["n"], case["L"],
                                         state["d_sfs"][p].data_ptr())
    rows(last, e.read_state_into(*state["bufs"][last]))
    state["sfs"].copy_(state["d_sfs"])
    out["sfs"] = state["sfs"]
    return out


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "sim":
        # per mutation-generation: its quarter of a Philox block, the draw and the selection step (about
        # forty operations); the state is made, and written once, on the way out
        theta = 4.0 * case["mu"] * case["N"] * case["L"]
        P = case["P"]
        held = P * theta * (math.log(2 * case["N"]) + 0.6)
        alive = held * (1 + 0.1 * case["compact"] / 25)
        return {"bytes": held * (4 * P + 16) * max(1, case["samples"]) + 1_632 * case["gens"],
                "flops": 40.0 * alive * P * case["gens"]}
    if kind == "spectra":
        gens = case["draws"] * case["reps"] * 0.525 * 2 * 3_900
        return {"bytes": case["draws"] * case["reps"] * 400.0 + 36 * gens, "flops": 40.0 * 2_000 * 8 * gens}
    if kind in ("sfs", "hist"):
        Nc = 2 * case["N"]
        if kind == "hist":
            return {"bytes": 4.0 * (case["M"] + Nc), "flops": 3.0 * case["M"]}
        return {"bytes": 4.0 * (case["M"] + case["n"]), "flops": 2.0 * min(case["M"], Nc) * (case["n"] + 1)}
    if kind == "joint":
        bins = (case["na"] + 1) * (case["nb"] + 1) * (case["nc"] + 1)
        return {"bytes": 4.0 * (case["M"] * (3 if case["nc"] else 2) + bins), "flops": 2.0 * case["M"] * bins}
    weights = sum(r * c for r, c in LAYERS)
    if kind == "forward":
        return {"bytes": case["batch"] * 4.0 * (6 + 99) + 2 * weights, "flops": 2.0 * case["batch"] * weights}
    if kind == "gradients":
        return {"bytes": case["batch"] * 4.0 * (6 + 99) + 8 * weights, "flops": 6.0 * case["batch"] * weights}
    if kind == "train":
        return {"bytes": case["steps"] * (case["batch"] * 4.0 * (6 + 99) + 28 * weights),
                "flops": case["steps"] * 6.0 * case["batch"] * weights}
    return {"bytes": case["count"] * 8.0 * (6 + 99) + 2 * weights, "flops": 2.0 * case["count"] * weights}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------
def _log_pmf(p, n):
    """log of the binomial(n, p) probabilities, [len(p)][n + 1], for 0 < p < 1."""
    k = torch.arange(n + 1, device=p.device, dtype=torch.float64)
    c = torch.lgamma(torch.tensor(n + 1.0, dtype=torch.float64, device=p.device)) - torch.lgamma(k + 1) - torch.lgamma(n - k + 1)
    return c + k * torch.log(p)[:, None] + (n - k) * torch.log1p(-p)[:, None]


def _pmf(p, n):
    p = p.double()
    inner = (p > 0) & (p < 1)
    out = torch.exp(_log_pmf(torch.where(inner, p, torch.full_like(p, 0.5)), n))
    point = torch.zeros((len(p), n + 1), dtype=torch.float64, device=p.device)
    point[:, 0] = (p <= 0).double()
    point[:, n] = (p >= 1).double()
    return torch.where(inner[:, None], out, point)


def _exact_sfs(row, n, L):
    values, counts = torch.unique(row, return_counts=True)
    inner = (values > 0) & (values < 1)
    lost = float(counts[~inner].sum()) + L - row.numel()
    values, counts = values[inner].double(), counts[inner].double()
    total = torch.zeros(n + 1, dtype=torch.float64, device=row.device)
    step = max(1, int(2e7 // (n + 1)))
    for a in range(0, len(values), step):
        total += counts[a:a + step] @ torch.exp(_log_pmf(values[a:a + step], n))
    total[0] += total[n] + lost
    return total[:n]


def _exact_joint(rows, case, L):
    shape = [case["na"] + 1, case["nb"] + 1] + ([case["nc"] + 1] if case["nc"] else [])
    total = torch.zeros((shape[0], math.prod(shape[1:])), dtype=torch.float64, device=rows[0].device)
    step = max(1, int(2e7 // math.prod(shape[1:])))
    for a in range(0, case["M"], step):
        part = _pmf(rows[1][a:a + step], case["nb"])
        if case["nc"]:
            part = (part[:, :, None] * _pmf(rows[2][a:a + step], case["nc"])[:, None, :]).flatten(1)
        total += _pmf(rows[0][a:a + step], case["na"]).T @ part
    total = total.reshape(shape)
    total[(0,) * len(shape)] += L - case["M"]
    return total


def _layers(vec, device):
    v, out, at = vec.to(device=device, dtype=torch.float64), [], 0
    for r, c in LAYERS:
        out.append((v[at:at + r * c].reshape(r, c), v[at + r * c:at + r * c + r]))
        at += r * c + r
    return out


def _net(x, layers):
    y = x.double()
    for i, (w, b) in enumerate(layers):
        y = y @ w.T + b
        if i < 4:
            y = torch.nn.functional.gelu(y, approximate="tanh")
    return y


def _gradients(x, t, layers):
    params = [q.detach().clone().requires_grad_(True) for pair in layers for q in pair]
    out = _net(x, list(zip(params[::2], params[1::2])))
    loss = ((out - t.double()) ** 2).mean()
    return params, torch.autograd.grad(loss, params), float(loss.detach())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sim", "spectra"):
        return None
    if kind == "sfs":
        return {"sfs": _exact_sfs(_row(case, seed), case["n"], float(20 * case["M"]))}
    if kind == "hist":
        Nc = 2 * case["N"]
        h = torch.bincount(torch.round(_row(case, seed).double() * Nc).long(), minlength=Nc + 1).double()
        h[0] += h[Nc] + 19 * case["M"]
        return {"hist": h[:Nc]}
    if kind == "joint":
        return {"joint": _exact_joint(_joint_rows(case, seed), case, float(20 * case["M"]))}
    if kind == "query":
        p = torch.from_numpy(_parameters(seed, case["count"])).cuda()
        low = torch.tensor([math.log(1e3), -100.0, 0.0, 0.0, -0.001, 0.05], dtype=torch.float64, device="cuda")
        high = torch.tensor([math.log(1e4), 10.0, 1.0, 0.5, 0.01, 1.0], dtype=torch.float64, device="cuda")
        x = 2 * (p - low) / (high - low) - 1
        g = [torch.asinh(v / 5.0) for v in (p[:, 1], low[1], high[1])]
        x[:, 1] = 2 * (g[0] - g[1]) / (g[2] - g[1]) - 1
        mean, std = (torch.from_numpy(v).cuda() for v in _scale(seed))
        q = torch.exp(_net(x, _layers(_weights(seed), "cuda")) * std + mean)
        return {"p": q / q.sum(1, keepdim=True), "routed": None}
    layers = _layers(_weights(seed), "cuda")
    if kind == "forward":
        return {"y": _net(_xy(seed, case["batch"])[0], layers)}
    x, t = _xy(seed, case["batch"] if kind == "gradients" else case["rows"])
    if kind == "gradients":
        _, grads, loss = _gradients(x, t, layers)
        return {"grads": torch.cat([g.flatten() for g in grads]), "loss": loss}
    # the same minibatches (drawn with replacement), cosine learning rate from 1e-3 to 1e-5 and Adam
    gen = _generator(seed)
    params = [q for pair in layers for q in pair]
    m = [torch.zeros_like(q) for q in params]
    v = [torch.zeros_like(q) for q in params]
    for s in range(case["steps"]):
        lr = 1e-5 + 0.5 * (1e-3 - 1e-5) * (1 + math.cos(math.pi * s / case["steps"]))
        idx = torch.randint(0, x.shape[0], (case["batch"],), device="cuda", generator=gen)
        _, grads, _ = _gradients(x[idx], t[idx], list(zip(params[::2], params[1::2])))
        for i, g in enumerate(grads):
            m[i] = 0.9 * m[i] + 0.1 * g
            v[i] = 0.999 * v[i] + 0.001 * g * g
            params[i] = params[i] - lr * (m[i] / (1 - 0.9 ** (s + 1))) / (torch.sqrt(v[i] / (1 - 0.999 ** (s + 1))) + 1e-8)
    return {"weights": torch.cat([q.flatten() for q in params])}
