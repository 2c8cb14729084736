"""Performance cases of the framework: what its users run, through its public
entry points, over the range of sizes that its configurations, tests and
benchmark cover.

  run    Simulation.run: a device-resident segment of simulated milliseconds
  step   Simulation.step once per millisecond, with stimulus and fired ids
         crossing the host boundary each time (a closed loop)
  batch  Batch.run: independent networks advanced together
  bptt   DifferentiableNetwork: a loss and its gradients (a training step)

Outputs of a simulation are its fire stream and the state it leaves (and
the weights where it learns and they fit a read each pass): integers and
fp32 bits that the framework reproduces exactly, so `exact` has nothing to
add for them.  Gradients have a 64-bit value, which `exact` computes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import nemosim_b200 as nb
from nemosim_b200.bptt import DifferentiableNetwork

f32 = np.float32

STDP_WINDOW = 20      # ms before and after a spike
RATE = 0.0066         # nominal spikes per neuron and ms of the random networks
TAU = 20.0            # ms, readout filter of the differentiable mode
MAX_SYNAPSES_DRAWN = 16_000_000


def listed():
    return [
        # the smallest unit of work: ten milliseconds of the 1000 x 100 example
        # network between two decisions of the host (launches and host path)
        {"name": "run_1k_10ms", "kind": "run", "neurons": 1000, "fanout": 100, "dmax": 20, "stdp": False, "ms": 10},
        # the same network for a simulated second, device-resident
        {"name": "run_1k_1s", "kind": "run", "neurons": 1000, "fanout": 100, "dmax": 20, "stdp": False, "ms": 1000},
        # a mid-sized, oddly sized network learning for 300 ms, reward every 100
        {"name": "run_10k_stdp", "kind": "run", "neurons": 10_007, "fanout": 100, "dmax": 20, "stdp": True, "ms": 300},
        # a large network without learning, 200 ms
        {"name": "run_100k", "kind": "run", "neurons": 100_000, "fanout": 100, "dmax": 32, "stdp": False, "ms": 200},
        # the benchmark network: 100k x 1000 with STDP, one reward period
        {"name": "run_100k_stdp", "kind": "run", "neurons": 100_000, "fanout": 1000, "dmax": 44, "stdp": True,
         "ms": 100},
        # mixed neuron types, heavy-tailed fan-out, scattered ids: 50k IF_curr_exp
        # + 50k Izhikevich + 10k Poisson sources
        {"name": "run_mixed_110k", "kind": "mixed", "neurons": 110_000, "fanout": 50, "dmax": 32, "ms": 200},
        # closed-loop control of a small learning network: 100 steps with a
        # firing stimulus each, then a reward and a look at the weights
        {"name": "step_1k_stdp", "kind": "step", "neurons": 1000, "fanout": 100, "dmax": 20, "stdp": True, "ms": 100,
         "fstim": 1, "istim": 0},
        # current injection into a mid-sized network, one millisecond a call
        {"name": "step_20k_current", "kind": "step", "neurons": 20_011, "fanout": 200, "dmax": 44, "stdp": False,
         "ms": 50, "fstim": 0, "istim": 128},
        # a parameter sweep: 24 networks of 1000 to 32000 neurons advanced together
        {"name": "batch_24", "kind": "batch", "networks": 24, "min_neurons": 1000, "max_neurons": 32_000,
         "min_fanout": 100, "max_fanout": 300, "dmax": 20, "ms": 200},
        # one training step of a small differentiable network (tests, prototyping)
        {"name": "bptt_256", "kind": "bptt", "neurons": 256, "fanout": 24, "dmax": 10, "ms": 80, "trials": 4,
         "readout": 32, "ckpt": 20, "double": True},
        # a training step at an odd size with float32 state
        {"name": "bptt_1k_float", "kind": "bptt", "neurons": 1021, "fanout": 100, "dmax": 10, "ms": 150, "trials": 7,
         "readout": 64, "ckpt": 50, "double": False},
        # the benchmark's training step: 4096 x 200, 500 ms, 16 trials, float64 state
        {"name": "bptt_4096", "kind": "bptt", "neurons": 4096, "fanout": 200, "dmax": 10, "ms": 500, "trials": 16,
         "readout": 256, "ckpt": 50, "double": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes spread over their logarithm."""
    kind = rng.choice(["run", "run", "step", "mixed", "batch", "bptt", "bptt"])
    if kind in ("run", "step"):
        neurons = _log_int(rng, 500, 100_000)
        fanout = min(_log_int(rng, 40, 1000), max(40, MAX_SYNAPSES_DRAWN // neurons))
        stdp = rng.random() < 0.5
        case = {"kind": kind, "neurons": neurons, "fanout": fanout, "dmax": rng.randint(10, 44), "stdp": stdp,
                "ms": _log_int(rng, 10, 500) if kind == "run" else _log_int(rng, 20, 120)}
        if kind == "step":
            case["fstim"] = rng.choice([0, 1, 5, 40])
            case["istim"] = rng.choice([0, 0, 7, 200])
        return case
    if kind == "mixed":
        return {"kind": "mixed", "neurons": _log_int(rng, 2000, 110_000), "fanout": rng.randint(20, 60),
                "dmax": rng.randint(10, 40), "ms": _log_int(rng, 20, 200)}
    if kind == "batch":
        return {"kind": "batch", "networks": rng.randint(3, 24), "min_neurons": 500,
                "max_neurons": _log_int(rng, 2000, 32_000), "min_fanout": 50, "max_fanout": rng.randint(60, 200),
                "dmax": rng.randint(5, 40), "ms": _log_int(rng, 20, 200)}
    trials, ms = rng.choice([1, 3, 4, 8, 13, 16]), _log_int(rng, 60, 300)
    neurons = _log_int(rng, 100, 3000)
    # float32 state only where rounding does not yet decide which neurons fire
    double = rng.random() < 0.75
    return {"kind": "bptt", "neurons": neurons, "fanout": _log_int(rng, 16, 200), "dmax": rng.randint(3, 10),
            "ms": ms if double else min(ms, 150), "trials": trials, "readout": max(8, neurons // rng.randint(4, 16)),
            "ckpt": rng.choice([20, 33, 50]), "double": double}


# ---------------------------------------------------------------------------
# networks

def _configuration(stdp):
    conf = nb.Configuration()
    if stdp:
        # exponential window, A+ = 0.1, A- = -0.12, weights within [-10, 10]
        dt = np.arange(1, STDP_WINDOW + 1, dtype=f32)
        conf.set_stdp_function((f32(0.1) * np.exp(-dt / f32(20.0))).astype(f32),
                               (f32(-0.12) * np.exp(-dt / f32(20.0))).astype(f32), -10.0, 10.0)
    return conf


def _generator_seed(seed, k=0):
    return (int(seed) * 2_654_435_761 + 40_503 * k + 12_345) % (1 << 32)


def _random_network(case, seed):
    return nb.example_random(case["neurons"], case["fanout"], case["dmax"], case["stdp"], _generator_seed(seed))


def _mixed_sizes(case):
    n_ps = case["neurons"] // 11
    n_if = (case["neurons"] - n_ps) // 2
    return n_if, case["neurons"] - n_ps - n_if, n_ps


def _mixed_network(case, seed):
    """IF_curr_exp, Izhikevich and 5 Hz Poisson neurons with interleaved ids,
    Pareto(1.5) out-degree, lognormal weights, a fifth of them inhibitory."""
    rng = np.random.default_rng(seed)
    net = nb.Network()
    tif, tiz, tps = (net.add_neuron_type(t) for t in ("IF_curr_exp", "Izhikevich", "PoissonSource"))
    n_if, n_iz, n_ps = _mixed_sizes(case)
    n = n_if + n_iz + n_ps
    ids = rng.permutation(n).astype(np.uint32)
    net.add_neuron(tif, ids[:n_if], -65.0, -65.0, 1.0, 20.0, 2.0, 5.0, 5.0, -50.0, 0.0, -65.0, 0.0, 0.0, 1000.0)
    r1, r2 = rng.random(n_iz, dtype=f32), rng.random(n_iz, dtype=f32)
    exc = rng.random(n_iz) < 0.8
    a = np.where(exc, f32(0.02), f32(0.02) + f32(0.08) * r1).astype(f32)
    b = np.where(exc, f32(0.2), f32(0.25) - f32(0.05) * r2).astype(f32)
    c = np.where(exc, f32(-65.0) + f32(15.0) * r1 * r1, f32(-65.0)).astype(f32)
    d = np.where(exc, f32(8.0) - f32(6.0) * r2 * r2, f32(2.0)).astype(f32)
    net.add_neuron(tiz, ids[n_if:n_if + n_iz], a, b, c, d, np.where(exc, f32(5.0), f32(2.0)).astype(f32),
                   (b * f32(-65.0)).astype(f32), f32(-65.0))
    net.add_neuron(tps, ids[n_if + n_iz:], f32(0.005))
    xm = case["fanout"] / 3.0
    deg = np.minimum((xm / rng.random(n) ** (1 / 1.5)).astype(np.int64), 1000)
    src = np.repeat(ids, deg).astype(np.uint32)
    tgt = ids[rng.integers(0, n, len(src))].astype(np.uint32)
    w = rng.lognormal(-1.0, 1.0, len(src)).astype(f32)
    w = np.where(rng.random(len(src)) < 0.2, -w, w).astype(f32)
    dly = rng.integers(1, case["dmax"] + 1, len(src)).astype(np.uint32)
    net.add_synapse(src, tgt, dly, w, np.zeros(len(src), np.uint8))
    return net


def _batch_sizes(case):
    """The sweep's sizes and noise: part of the case, not of its inputs."""
    k = case["networks"]
    rng = np.random.default_rng(k)
    return (rng.integers(case["min_neurons"], case["max_neurons"] + 1, k),
            rng.integers(case["min_fanout"], case["max_fanout"] + 1, k), rng.uniform(2.0, 8.0, k))


def _bptt_inputs(case, seed):
    """Structure and tensors of a differentiable network: 80/20 Izhikevich
    neurons, normal weights, Gaussian input noise, and as targets the
    filtered trains of 10 Hz Poisson teachers."""
    dev = torch.device("cuda", torch.cuda.current_device())
    N, F, T, B, R = (case[k] for k in ("neurons", "fanout", "ms", "trials", "readout"))
    rng = np.random.default_rng(seed)
    exc = np.arange(N) < int(0.8 * N)
    r1, r2 = rng.random(N, dtype=f32), rng.random(N, dtype=f32)
    s = {"a": np.where(exc, 0.02, 0.02 + 0.08 * r1), "b": np.where(exc, 0.2, 0.25 - 0.05 * r2),
         "c": np.where(exc, -65.0 + 15.0 * r1 * r1, -65.0), "d": np.where(exc, 8.0 - 6.0 * r2 * r2, 2.0),
         "weight": rng.normal(0.0, 0.5 / np.sqrt(F), N * F)}
    s = {k: v.astype(f32) for k, v in s.items()}
    s["source"] = np.repeat(np.arange(N, dtype=np.uint32), F)
    s["target"] = rng.integers(0, N, N * F, dtype=np.uint32)
    s["delay"] = rng.integers(1, case["dmax"] + 1, N * F, dtype=np.uint32)
    g = torch.Generator(device=dev).manual_seed(int(seed))
    noise = 5.0 * torch.randn((T, B, N), generator=g, device=dev)
    spikes = (torch.rand((T, B, R), generator=g, device=dev) < 0.01).float()
    target, r, alpha = torch.empty_like(spikes), torch.zeros((B, R), device=dev), math.exp(-1.0 / TAU)
    for t in range(T):
        r = alpha * r + spikes[t]
        target[t] = r
    return s, noise, target


# ---------------------------------------------------------------------------
# a case's state and one pass

def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind in ("run", "step"):
        state["sim"] = nb.Simulation(_random_network(case, seed), _configuration(case["stdp"]))
        state["types"] = [(0, 2, case["neurons"])]
        if kind == "step":
            rng = np.random.default_rng(seed)
            n = case["neurons"]
            state["fstim"] = [rng.choice(n, case["fstim"], replace=False).tolist() for _ in range(case["ms"])]
            state["istim"] = [list(zip(rng.choice(n, case["istim"], replace=False).tolist(),
                                       rng.uniform(0.0, 8.0, case["istim"]).tolist())) for _ in range(case["ms"])]
    elif kind == "mixed":
        state["sim"] = nb.Simulation(_mixed_network(case, seed), _configuration(False))
        n_if, n_iz, _ = _mixed_sizes(case)
        state["types"] = [(0, 4, n_if), (1, 2, n_iz)]
    elif kind == "batch":
        sizes, fanouts, sigmas = _batch_sizes(case)
        nets = [nb.example_random(int(n), int(f), case["dmax"], False, _generator_seed(seed, k), float(s), 2.0)
                for k, (n, f, s) in enumerate(zip(sizes, fanouts, sigmas))]
        state["sim"] = nb.Batch(nets, _configuration(False))
        state["sizes"] = [int(n) for n in sizes]
    else:
        s, noise, target = _bptt_inputs(case, seed)
        net = DifferentiableNetwork(**s)
        state["model"] = net.model(case["trials"], case["ms"], case["readout"], case["ckpt"],
                                   state_dtype=torch.float64 if case["double"] else torch.float32)
        state["leaves"] = net.tensors(noise.device)
        state["noise"], state["target"] = noise, target
    if kind != "bptt":
        neurons = sum(state["sizes"]) if kind == "batch" else case["neurons"]
        state["ids"], state["stored"] = np.zeros(_max_ids(case, neurons), np.uint32), 0
    return state


def _max_ids(case, neurons):
    return case["ms"] * max(64, neurons // 8)


def _keep(state, ids):
    """The fired ids in the program's own buffer of fixed size, zeros after
    the last."""
    buf, before = state["ids"], state["stored"]
    buf[:len(ids)] = ids
    buf[len(ids):before] = 0
    state["stored"] = len(ids)
    return buf


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "bptt":
        W, a, b = state["leaves"]
        loss = state["model"].loss(W, a, b, state["noise"], state["target"])
        return (loss.detach(),) + torch.autograd.grad(loss, (W, a, b))
    sim = state["sim"]
    if kind == "batch":
        counts, events, ids = sim.run(case["ms"], max_ids=len(state["ids"]))
        return counts, events, _keep(state, ids), [sim.type_state(k, 0, 2, n) for k, n in enumerate(state["sizes"])]
    if kind == "step":
        fired = [sim.step(f, i) for f, i in zip(state["fstim"], state["istim"])]
        out = [np.array([len(f) for f in fired]), _keep(state, [i for f in fired for i in f])]
        if case["stdp"]:
            sim.apply_stdp(1.0)
    else:
        period = 100 if case.get("stdp") else 0
        counts, events, ids = sim.run(case["ms"], period, 1.0, max_ids=len(state["ids"]))
        out = [counts, events, _keep(state, ids)]
    out += [sim.type_state(*t) for t in state["types"]]
    # the weights of the largest networks are read at the end of a program,
    # not once a pass
    if case.get("stdp") and case["neurons"] * case["fanout"] <= 2_000_000:
        out.append(sim.weights_fx(case["neurons"] * case["fanout"]))
    return out


# ---------------------------------------------------------------------------
# what one pass cannot do without

def work(case):
    ms = case["ms"]
    if case["kind"] == "bptt":
        N, T, B, M = case["neurons"], ms, case["trials"], case["neurons"] * case["fanout"]
        # noise and targets in, weights and parameters in, gradients out
        nbytes = 4 * T * B * (N + case["readout"]) + 4 * M * (2 + 2) + 4 * 6 * N
        # four sub-steps forward (18 flops each) and their adjoint (35), twice
        # the sub-steps for the adjoint's own replay, a multiply-add per synapse
        # for each input adjoint, and one per arriving spike for the inputs and
        # for the weight gradients
        flops = T * B * (N * 4 * (18 + 18 + 35) + 2 * M + 2 * 2 * M * RATE)
        return {"bytes": nbytes, "flops": flops}
    if case["kind"] == "batch":
        N = case["networks"] * (case["min_neurons"] + case["max_neurons"]) / 2
        fanout = (case["min_fanout"] + case["max_fanout"]) / 2
    else:
        N, fanout = case["neurons"], case["fanout"]
    events = N * fanout * RATE * ms
    # neurons in and out once (parameters, state, RNG words), 8 bytes per
    # synaptic event, 4 per fired id
    nbytes = N * 60 + events * 8 + N * RATE * ms * 4
    flops = N * ms * 60 + events
    if case.get("stdp"):
        # incoming plastic synapses of each spike: source, history and
        # accumulator; 20 bytes per plastic synapse and reward
        plastic = 0.8 * N * fanout
        nbytes += 12 * plastic * RATE * ms + 20 * plastic * max(1, ms // 100)
        flops += plastic * RATE * ms * 4
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values

def exact(case, seed):
    """Loss and gradients in float64, the adjoint written out in dense
    matrices.  None for simulations (their outputs are whole numbers, and
    fp32 bits whose rounding is part of the result) and for float32 state,
    where rounding decides which neurons fire."""
    if case["kind"] != "bptt" or not case["double"]:
        return None
    s, noise, target = _bptt_inputs(case, seed)
    dev = noise.device
    N, T, B, R, D = (case[k] for k in ("neurons", "ms", "trials", "readout", "dmax"))
    a, b, c, d = (torch.tensor(s[k], device=dev).double() for k in "abcd")
    w = torch.tensor(s["weight"], device=dev).double()
    src, tgt, dly = (torch.tensor(s[k].astype(np.int64), device=dev) for k in ("source", "target", "delay"))
    # dense[d - 1, j, n]: the weights from j to n with delay d
    dense = torch.zeros((D, N, N), dtype=torch.float64, device=dev)
    dense.index_put_((dly - 1, src, tgt), w, accumulate=True)
    noise, target = noise.double(), target.double()
    alpha = math.exp(-1.0 / TAU)
    # spikes and input adjoints, padded by D ms of silence on either side
    S = torch.zeros((T + 2 * D, B, N), dtype=torch.float64, device=dev)
    lamI = torch.zeros_like(S)
    v, u = torch.full((B, N), -65.0, dtype=torch.float64, device=dev), b * torch.full_like(noise[0], -65.0)
    r, rs, trace, loss = torch.zeros_like(target[0]), [], [], 0.0
    for t in range(T):
        past = S[t:t + D].flip(0)  # S(t - 1) ... S(t - D)
        I = torch.bmm(past, dense).sum(0) + noise[t]
        total = torch.zeros_like(v)
        steps = []
        for _ in range(4):
            v1 = v + 0.25 * (0.04 * v * v + 5.0 * v + 140.0 - u + I)
            u1 = u + 0.25 * a * (b * v1 - u)
            sp = (v1 >= 30.0).double()
            steps.append((v, u, v1, sp))
            v, u = v1 + sp * (c - v1), u1 + sp * d
            total = total + sp
        trace.append(torch.stack([torch.stack(x) for x in steps]))
        S[t + D] = total
        r = alpha * r + total[:, :R]
        rs.append(r - target[t])
        loss = loss + (rs[-1] ** 2).sum()
    scale = 1.0 / (T * R * B)
    lv, lu, lr = torch.zeros_like(v), torch.zeros_like(v), torch.zeros_like(r)
    ga, gb = torch.zeros_like(v), torch.zeros_like(v)
    back = dense.transpose(1, 2)
    for t in reversed(range(T)):
        lr = 2.0 * scale * rs[t] + alpha * lr
        ls = torch.bmm(lamI[t + D + 1:t + 2 * D + 1], back).sum(0)
        ls[:, :R] += lr
        li = torch.zeros_like(v)
        for v0, u0, v1, sp in trace[t].flip(0):
            lsp = ls + lv * (c - v1) + lu * d
            q = 1.0 + 10.0 * (v1 - 30.0).abs()
            lv1 = lv * (1.0 - sp) + lsp * (5.0 / (q * q)) + lu * 0.25 * a * b
            ga += lu * 0.25 * (b * v1 - u0)
            gb += lu * 0.25 * a * v1
            lu = lu * (1.0 - 0.25 * a) - 0.25 * lv1
            lv = lv1 * (1.0 + 0.25 * (0.08 * v0 + 5.0))
            li += 0.25 * lv1
        lamI[t + D] = li
    gW = torch.empty_like(w)
    flat = S[D:D + T].reshape(T * B, N)
    for k in range(1, D + 1):
        # sum over t, b of S_j(t) lamI_n(t + k)
        full = flat.t() @ lamI[D + k:D + k + T].reshape(T * B, N)
        at = dly == k
        gW[at] = full[src[at], tgt[at]]
    return loss * scale, gW, ga.sum(0), (gb + lu * -65.0).sum(0)
