"""Performance cases: the work that programs give this package, each through the
entry point that they call.

`listed()` names the cases, `draw(rng)` gives further ones of the same families
and ranges, `prepare(case, seed)` builds what a program holds before the call
(inputs from the seed, prepared graphs, kept plans), `run(state)` is one pass,
`work(case)` the bytes and operations that a pass cannot do without, and
`exact(case, seed)` the float64 values of its computed outputs where they have
any.

Graph families, in the sizes and distributions of the package's workloads:
  reg  3-regular, +-1 couplings (integer weights, sparse)
  er   G(n, 0.5), unit weights (integer weights, dense)
  gnp  G(n, 0.1), weights uniform in (0, 1] (float32)
  sk   complete graph, J ~ N(0, 1) / sqrt(n) (float32)
"""

from __future__ import annotations

import importlib
import math

import numpy as np
import torch

from pyqrackising_b200 import learned, maxcut_tfim, spin_glass_solver, workloads
from pyqrackising_b200 import device as D
from pyqrackising_b200.batch import BatchedSearch, BatchedSolver

# the package exports the drop-in functions under their modules' names
sampler = importlib.import_module("pyqrackising_b200.maxcut_tfim")

GPU = "cuda"


def listed():
    return [
        # the smallest call: the drop-in solver on the 64-node README instance from a given
        # partition, host array in, partition out - launches and host round trips count
        {"name": "solve_reg64", "do": "solve", "graph": "reg", "n": 64, "host": True},
        # the drop-in solver's loop (descent, pair pass, Gray search) at the largest dense size
        # in use, a float32 spin glass already on the device
        {"name": "solve_sk8192", "do": "solve", "graph": "sk", "n": 8192, "host": False},
        # the drop-in MAXCUT call with its default quality: Hamming-weight distribution,
        # sampled batches, scoring, until a batch brings nothing better
        {"name": "maxcut_er1024", "do": "maxcut", "graph": "er", "n": 1024, "quality": 6, "host": True},
        # one sampling round on a sparse graph (distribution and candidates), the seed of the
        # solver on 3-regular instances
        {"name": "sample_reg2048", "do": "sample", "graph": "reg", "n": 2048, "quality": 6, "shots": 16384},
        # the batch that the MAXCUT call scores per round at quality 6 on 2048 nodes: exact
        # integer weights, the largest ordinary batch
        {"name": "score_er2048", "do": "score", "graph": "er", "n": 2048, "shots": 65536, "spin": False},
        # scoring of a float32 spin glass at the largest dense size
        {"name": "score_sk8192", "do": "score", "graph": "sk", "n": 8192, "shots": 4096, "spin": True},
        # an odd node count and a small ragged batch of float32 weights: launch-bound scoring
        {"name": "score_gnp777", "do": "score", "graph": "gnp", "n": 777, "shots": 3001, "spin": False},
        # one exact pass over all pairs from a single-flip local optimum (between descents)
        {"name": "double_sk8192", "do": "double", "graph": "sk", "n": 8192, "spin": True},
        # low-latency ascent of a few starts, one thread-block cluster each
        {"name": "ascent_sk8192", "do": "ascent", "graph": "sk", "n": 8192, "tasks": 32, "cluster": 8},
        # the batched service: many small uneven graphs of both weight kinds, many starts each
        {"name": "batch_uneven", "do": "batch", "graphs": 192, "lo": 64, "hi": 1024, "starts": 64},
        # iterated search (ascent, kicks, ascent) of many starts on one large odd-sized graph
        {"name": "iterate_sk5999", "do": "iterate", "graph": "sk", "n": 5999, "tasks": 592, "rounds": 2, "kick": 64},
        # forward and backward of one training example of the proposal network
        {"name": "learn_gnp1024", "do": "learn", "graph": "gnp", "n": 1024},
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    do = rng.choice(["solve", "maxcut", "sample", "score", "score", "double", "ascent", "batch", "iterate", "learn"])
    kind = rng.choice(["reg", "er", "gnp", "sk"])
    if do == "solve":
        c = {"do": do, "graph": kind, "n": _log(rng, 24, 6000), "host": rng.random() < 0.5}
    elif do == "maxcut":
        c = {"do": do, "graph": kind, "n": _log(rng, 32, 900), "quality": rng.randint(2, 6), "host": True}
    elif do == "sample":
        c = {"do": do, "graph": kind, "n": _log(rng, 32, 1536), "quality": rng.randint(2, 6), "shots": _log(rng, 64, 8192)}
    elif do == "score":
        n = _log(rng, 64, 8192)
        c = {"do": do, "graph": kind, "n": n, "shots": _log(rng, 33, min(65536, (1 << 37) // (n * n))), "spin": rng.random() < 0.5}
    elif do == "double":
        c = {"do": do, "graph": kind, "n": _log(rng, 64, 8000), "spin": rng.random() < 0.5}
    elif do == "ascent":
        c = {"do": do, "graph": kind, "n": _log(rng, 512, 8000), "tasks": rng.randint(1, 32), "cluster": rng.choice([2, 4, 8, 16])}
        if c["n"] > 4000:
            c["cluster"] = max(4, c["cluster"])
    elif do == "batch":
        hi = _log(rng, 128, 1024)
        c = {"do": do, "graphs": rng.randint(8, 160), "lo": 64, "hi": hi, "starts": rng.randint(8, 64)}
    elif do == "iterate":
        c = {"do": do, "graph": kind, "n": _log(rng, 256, 5600), "tasks": _log(rng, 16, 592), "rounds": rng.randint(1, 3), "kick": rng.randint(4, 64)}
    else:
        c = {"do": do, "graph": kind, "n": _log(rng, 128, 1500)}
    if c.get("graph") == "reg":
        c["n"] += c["n"] % 2  # a 3-regular graph has an even node count
    return c


# ------------------------------------------------------------------------------------
# inputs


def _generator(seed):
    g = torch.Generator(device=GPU)
    g.manual_seed(int(seed))
    return g


def _matrix(kind, n, seed):
    """Dense symmetric float32 couplings with a zero diagonal, on the device."""
    if kind == "reg":
        return torch.from_numpy(workloads.regular_pm1_np(n, seed)).to(GPU)
    g = _generator(seed)
    if kind == "er":
        w = (torch.rand(n, n, generator=g, device=GPU) < 0.5).float()
    elif kind == "gnp":
        w = torch.where(torch.rand(n, n, generator=g, device=GPU) < 0.1,
                        1.0 - torch.rand(n, n, generator=g, device=GPU), 0.0)
    else:
        w = torch.randn(n, n, generator=g, device=GPU) / math.sqrt(n)
    w = torch.triu(w, 1)
    return (w + w.T).contiguous()


def _bits(rows, n, seed):
    return (torch.rand(rows, n, generator=_generator(seed + 7919), device=GPU) < 0.5).to(torch.uint8)


def _mpe():
    return D.max_gpu_proc_elem(D.default_device())


def _batch_graphs(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i, n in enumerate(rng.integers(case["lo"], case["hi"] + 1, size=case["graphs"])):
        n, s = int(n), int(rng.integers(1 << 30))
        out.append(_matrix("gnp", n, s) if i % 2 else _matrix("reg", n + n % 2 if n < case["hi"] else n - n % 2, s))
    return out


HID, FEAT, LAYERS = learned.HID, learned.FEAT, learned.LAYERS


def _net_params(seed):
    """Float32 parameters of the proposal network, in its storage order."""
    rng = np.random.default_rng(seed)
    parts = [rng.standard_normal(FEAT * HID) * math.sqrt(2.0 / FEAT), np.full(HID, 0.01)]
    for _ in range(LAYERS):
        parts += [rng.standard_normal(2 * HID * HID) * math.sqrt(1.0 / HID), np.full(HID, 0.01)]
    parts += [rng.standard_normal(HID) * math.sqrt(1.0 / HID), np.full(1, 0.01)]
    return np.concatenate(parts).astype(np.float32)


def _net_target(n, seed):
    """Uniform over the nodes where two optima differ (about a sixteenth of them)."""
    t = (torch.rand(n, generator=_generator(seed + 104729), device=GPU) < 1 / 16).float()
    t[0] = 1.0
    return t / t.sum()


def prepare(case, seed):
    do = case["do"]
    if do == "batch":
        solver = BatchedSolver([D.DeviceGraph(w) for w in _batch_graphs(case, seed)], case["starts"], True, seed=seed)
        solver.set_starts(seed)
        solver.autotune(reps=1)
        solver.capture()
        return case, solver
    n = case["n"]
    W = _matrix(case["graph"], n, seed)
    if do in ("solve", "maxcut"):
        G = W.cpu().numpy() if case["host"] else W
        guess = "".join("1" if b else "0" for b in _bits(1, n, seed)[0].tolist())
        return case, G, guess, seed
    dg = D.DeviceGraph(W)
    if do == "sample":
        sampler.row_lists(dg)  # built once per prepared graph
        return case, dg, seed
    if do == "score":
        words = dg.pack(_bits(case["shots"], n, seed))
        return case, dg, words, D.geometry(case["shots"], case["shots"], _mpe())
    if do == "double":
        words = dg.pack(_bits(1, n, seed))
        _, g64 = dg.gains(words)
        geo = D.geometry(min(D.WORK_GROUP_MULTIPLE, n), n, _mpe())
        dg.single_descent(words, g64, case["spin"], *geo, 4 * n)
        return case, dg, words, g64, geo
    if do == "learn":
        net = learned.ProposalNet(params=_net_params(seed))
        ctx = learned.GraphContext(dg)
        return case, net, ctx, dg.pack(_bits(1, n, seed)), _net_target(n, seed)
    bs = BatchedSearch([dg])
    tg = np.zeros(case["tasks"], dtype=np.int32)
    words = bs.random_states(tg, seed)
    if do == "iterate":  # the task list kept on the device, as BatchedSolver keeps it
        tg = torch.from_numpy(tg).to(GPU)
    return case, bs, tg, words, seed


# ------------------------------------------------------------------------------------
# one pass


def run(state):
    case, do = state[0], state[0]["do"]
    if do == "solve":
        _, G, guess, _ = state
        bits, cut, _, energy = spin_glass_solver(G, best_guess=guess)
        return {"bits": np.frombuffer(bits.encode(), dtype=np.uint8), "cut": cut, "energy": energy}
    if do == "maxcut":
        _, G, _, seed = state
        sampler.set_seed(seed)
        bits, cut, _ = maxcut_tfim(G, quality=case["quality"])
        return {"bits": np.frombuffer(bits.encode(), dtype=np.uint8), "cut": cut}
    if do == "sample":
        _, dg, seed = state
        J, degrees, cum = sampler.hamming_cdf(dg, case["quality"], 8.0, 8.0)
        words = sampler.sample_batch(dg, cum, case["shots"], 5.0, seed, 0)
        return {"J": J, "degrees": degrees, "cum": cum, "words": words}
    if do == "score":
        _, dg, words, geo = state
        e, be, bi = dg.calculate_cut(words, case["shots"], case["spin"], *geo)
        return {"values": e, "best": be, "index": bi}
    if do == "double":
        _, dg, words, g64, geo = state
        be, bi = dg.double_bit_flips(words, g64, case["spin"], *geo)
        return {"best": be, "index": bi}
    if do == "ascent":
        _, bs, tg, words, _ = state
        values, states, flips, status = bs.cluster_ascent(tg, words, True, cluster_size=case["cluster"])
        return {"values": values, "states": states, "flips": flips, "status": status}
    if do == "iterate":
        _, bs, tg, words, seed = state
        values, states, flips, status = bs.run(tg, words, True, rounds=case["rounds"], kick=case["kick"], seed=seed)
        return {"values": values, "states": states, "flips": flips, "status": status}
    if do == "batch":
        _, solver = state
        solver.step()
        return [grp["out"] for grp in solver.groups]
    _, net, ctx, words, target = state
    net.zero_grad()
    logits, cache = net.forward(ctx, ctx.features(words))
    loss, dlogits, _ = net.loss_grad(logits, target)
    net.backward(ctx, cache, dlogits)
    return {"logits": logits, "loss": loss, "gradient": net.g}


# ------------------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    do = case["do"]
    if do == "batch":
        mean = (case["lo"] + case["hi"]) / 2
        tasks = case["graphs"] * case["starts"]
        # per task: its starting fields and about half a flip per node, each reading a row
        return {"bytes": case["graphs"] * mean * mean * 2.5 + tasks * (mean / 4 + 8), "flops": tasks * 2.0 * mean * mean}
    n = case["n"]
    wb = 1 if case["graph"] in ("reg", "er") else 4
    if do == "solve":
        # W in, about half a row update per node, one pass over all pairs
        return {"bytes": 4.0 * n * n + wb * n * n / 2, "flops": 4.0 * n * n}
    if do == "maxcut":
        # two rounds: n/2 picks of a row update each, then x^T W x over the pairs
        shots = (n << case["quality"]) / 2
        return {"bytes": 4.0 * n * n + 2 * shots * n / 8, "flops": 2 * shots * 2.0 * n * n}
    if do == "sample":
        row = 3 if case["graph"] == "reg" else n
        return {"bytes": 4.0 * n * n + case["shots"] * n / 8, "flops": case["shots"] * (n / 2) * 2.0 * (row + math.log2(n))}
    if do == "score":
        planes = 1 if wb == 1 else 4
        return {"bytes": float(n * n * planes) + case["shots"] * (n / 8 + 4), "flops": float(case["shots"]) * n * n * planes}
    if do == "double":
        return {"bytes": wb * n * (n - 1) / 2 + 8.0 * n, "flops": 1.5 * n * n}
    if do in ("ascent", "iterate"):
        flips = 0.6 * n + case.get("rounds", 0) * case.get("kick", 0) * 2
        return {"bytes": float(wb) * n * n + case["tasks"] * (n / 4 + 8), "flops": case["tasks"] * (2.0 * n * n + 2.0 * flips * n)}
    params = FEAT * HID + LAYERS * 2 * HID * HID
    return {"bytes": 2.0 * n * n + 4.0 * n * HID * LAYERS, "flops": 4.0 * n * n * HID * LAYERS + 6.0 * n * params}


# ------------------------------------------------------------------------------------
# float64 values


def _exact_scores(case, seed):
    n, shots, spin = case["n"], case["shots"], case["spin"]
    W = _matrix(case["graph"], n, seed).double()
    X = _bits(shots, n, seed)
    out = torch.empty(shots, dtype=torch.float64, device=GPU)
    for lo in range(0, shots, 4096):
        x = 2.0 * X[lo:lo + 4096].double() - 1.0
        q = ((x @ W) * x).sum(1)
        out[lo:lo + 4096] = -q / 2 if spin else (W.sum() - q) / 4
    return {"values": out, "best": out.max().reshape(1), "index": None}


def _exact_cdf(case, seed):
    """The Hamming-weight distribution of the TFIM sampler: per time step and node the
    magnetisation envelope at t and t - dt, both normalised, their differences
    accumulated on the binomial start, then the cumulative sum over 1 .. n-1."""
    n, quality, h, tot = case["n"], case["quality"], 8.0, 8.0
    eps = 1.1920928955078125e-07
    W = _matrix(case["graph"], n, seed)
    val = (W - W.min()).double()
    edge = val > eps
    degrees = edge.sum(1)
    J = torch.where(degrees > 0, -(val * edge).sum(1) / degrees.clamp(min=1), 0.0)
    k = torch.arange(n + 1, dtype=torch.float64, device=GPU)
    half = n / 2.0
    acc = np.zeros(n + 1)
    comb, norm = 1, 0
    for q in range(n >> 1):
        norm += math.comb(n, q) << 1
    if n & 1:
        norm += math.comb(n, n >> 1)
    for q in range(n >> 1):
        acc[q] = acc[n - q] = comb / norm
        comb = math.comb(n, q + 1)
    if n & 1:
        acc[n >> 1] = comb / norm
    acc = torch.from_numpy(acc).to(GPU)
    live = J.abs() >= eps
    Jl, z = J[live], degrees[live].double()
    zJ = z * Jl
    quarter = torch.where(Jl > 0, math.pi / 2, -math.pi / 2)
    theta = torch.where(zJ.abs() < eps, quarter, torch.asin((h / zJ).clamp(-1, 1)))
    steps = 1 << quality
    for step in range(1, steps):
        t, dt = step * (tot / steps), tot / steps
        ht = h * (tot - t)
        theta_c = torch.where(zJ.abs() < eps, quarter, torch.asin((ht / zJ).clamp(-1, 1)))
        for sign, tt in ((1.0, t), (-1.0, t - dt)):
            p = torch.exp2((Jl / ht).abs() - 1.0) * (1.0 + torch.sin(theta - theta_c) * torch.cos(1.5 * math.pi * Jl * tt + theta) / (1.0 + math.sqrt(tt))) - 0.5
            bias = torch.exp2(-(p / (n + 1))[:, None] * (k + 1.0)[None, :])
            env = bias / bias.sum(1, keepdim=True) * torch.exp(-(k - half).abs() / max(tt, 1e-9))[None, :]
            total = env.sum(1, keepdim=True)
            delta = torch.zeros(n + 1, dtype=torch.float64, device=GPU)
            delta[n // 2] = 1.0
            acc += sign * torch.where(total > 0, env / total, delta[None, :]).sum(0)
    cum = torch.cumsum(acc[1:n] / acc[1:n].sum(), 0)
    cum[-1] = 1.0
    return {"J": J, "degrees": None, "cum": cum, "words": None}


def _exact_logits(case, seed):
    """The proposal network's logits and loss in float64 from the float32 parameters."""
    n = case["n"]
    W = _matrix(case["graph"], n, seed).double()
    x = 2.0 * _bits(1, n, seed)[0].double() - 1.0
    s = W.abs().sum(1)
    A = W / torch.sqrt(s[:, None].clamp(min=1e-30) * s[None, :].clamp(min=1e-30))
    p = torch.from_numpy(_net_params(seed)).to(GPU).double()
    at = 0

    def take(*shape):
        nonlocal at
        size = math.prod(shape)
        out = p[at:at + size].reshape(shape)
        at += size
        return out

    F = torch.stack([x, x * (W @ x) / s.clamp(min=1e-30), s / s.mean(), torch.ones_like(s)], 1)
    H = torch.relu(F @ take(FEAT, HID) + take(HID))
    for _ in range(LAYERS):
        H = torch.relu(torch.cat([H, A @ H], 1) @ take(2 * HID, HID) + take(HID))
    logits = H @ take(HID) + take(1)
    loss = -(_net_target(n, seed).double() * torch.log_softmax(logits, 0)).sum().reshape(1)
    return {"logits": logits, "loss": loss, "gradient": None}


def exact(case, seed):
    if case["do"] == "score":
        return _exact_scores(case, seed)
    if case["do"] == "sample":
        return _exact_cdf(case, seed)
    if case["do"] == "learn":
        return _exact_logits(case, seed)
    return None  # partitions and the values of the states that a search ends in
