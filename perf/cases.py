"""Performance cases of the simulation backend: what a user's program does through the public
entry points, at sizes from the smallest networks to the configured benchmarks.

A case is a dict of plain values.  `prepare` builds what such a program holds before it starts
simulating (a finalized network with a device checkpoint, a multicompartment batch, a
surrogate with its data), `run` is one pass: back to the checkpoint, `steps` time steps, the
whole updated state.  The networks of one program share one CUDA stream, and neuron state is
read where it lives, through `Network.state_ptr` as tensors.

Launch shapes and step forms are the library's own rules or an explicit option of `Network`;
nothing is autotuned here, because two tunings of one program may keep different step forms,
which round float32 sums differently.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from brian2cuda_b200 import models
from brian2cuda_b200.network import LIF, HinesParams, Network
from brian2cuda_b200.surrogate import GatingSurrogate

DT = 1e-4            # s, the networks' time step
HINES_DT = 25e-6     # s, the multicompartment batch's
MON = 1 << 25        # spike monitor entries: more than every pass of a program here records
CUBA_INDEGREE = 80   # synapses per neuron of the CUBA network at its configured 4000 neurons
P_CONNECT = 0.02     # connection probability of the COBAHH-shaped networks
DELAYS = (1, 50)     # their delays in steps

HH_VARS = ("v", "m", "h", "n", "ge", "gi", "lastspike")
LIF_VARS = ("v", "ge", "gi", "lastspike")


def listed():
    return [
        # CUBA (examples/cuba.py) at the size of a first experiment, on the option for small
        # networks: a few microseconds per step, all latency
        {"name": "cuba_700_small", "kind": "cuba", "n": 700, "dtype": "float64", "small": True,
         "steps": 500},
        # CUBA as configured: 4000 LIF neurons, float64, no delays, the default form
        {"name": "cuba_4000", "kind": "cuba", "n": 4000, "dtype": "float64", "small": False,
         "steps": 1000},
        # the same network scaled up, float32, with axonal delays
        {"name": "cuba_delays_150k", "kind": "cuba_delays", "n": 150_001, "dtype": "float32",
         "steps": 500},
        # COBAHH (examples/cobahh.py) of ordinary, odd size in Brian2's default precision
        {"name": "cobahh_8001_f64", "kind": "cobahh", "n": 8001, "dtype": "float64",
         "one_launch": False, "steps": 1000},
        # COBAHH as configured (1e5 neurons, 2e8 synapses, delays 1-50), in the step form that
        # a tuned program keeps for it; the window holds bursts and the quiet between them
        {"name": "cobahh_100k", "kind": "cobahh", "n": 100_000, "dtype": "float32",
         "one_launch": True, "steps": 2000},
        # a parameter sweep: independent COBAHH instances of uneven sizes in one network
        {"name": "batched_40", "kind": "batched", "instances": 40, "steps": 300},
        # spike propagation at high load as configured (~6e6 events per step)
        {"name": "propagation_100k", "kind": "propagation", "n_in": 100_000, "n_out": 100_000,
         "rate": 300.0, "steps": 200},
        # STDP as configured: 1e4 Poisson inputs, all-to-all onto 1e3 LIF neurons, float32
        {"name": "stdp_10k_1k_f32", "kind": "stdp", "n_in": 10_000, "n_out": 1000,
         "dtype": "float32", "replay": False, "delay": 0, "steps": 500},
        # STDP of ordinary, odd size in float64: recorded spike trains with a delay
        {"name": "stdp_3001_257_f64", "kind": "stdp", "n_in": 3001, "n_out": 257,
         "dtype": "float64", "replay": True, "delay": 8, "steps": 300},
        # the multicompartment batch as configured: 1024 morphologies of 200-1000 compartments
        {"name": "hines_1024_f32", "kind": "hines", "neurons": 1024, "comps": 1000,
         "channels": "float32", "steps": 500},
        # a small batch of small morphologies with float64 channels: fewer neurons than SMs
        {"name": "hines_61_f64", "kind": "hines", "neurons": 61, "comps": 400,
         "channels": "float64", "steps": 200},
        # the gating surrogate on a data set: predictions, loss and gradient (the two halves
        # of its training step, forward and backward)
        {"name": "surrogate_1m", "kind": "surrogate", "rows": 1_000_037},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("cuba", "cuba_delays", "cobahh", "batched", "propagation", "stdp",
                       "hines", "surrogate"))
    if kind == "cuba":
        n = log_int(300, 20_000)
        return {"kind": kind, "n": n, "dtype": rng.choice(("float64", "float32")),
                "small": n <= 2000, "steps": 500}
    if kind == "cuba_delays":
        return {"kind": kind, "n": log_int(5000, 150_000),
                "dtype": rng.choice(("float64", "float32")), "steps": 500}
    if kind == "cobahh":
        dtype = rng.choice(("float32", "float32", "float64"))
        return {"kind": kind, "n": log_int(2000, 100_000 if dtype == "float32" else 30_000),
                "dtype": dtype, "one_launch": rng.random() < 0.5, "steps": 1000}
    if kind == "batched":
        return {"kind": kind, "instances": log_int(4, 40), "steps": 200}
    if kind == "propagation":
        return {"kind": kind, "n_in": log_int(10_000, 100_000), "n_out": log_int(10_000, 100_000),
                "rate": round(math.exp(rng.uniform(math.log(30.0), math.log(300.0))), 1),
                "steps": 150}
    if kind == "stdp":
        replay = rng.random() < 0.5
        return {"kind": kind, "n_in": log_int(500, 10_000 if not replay else 4000),
                "n_out": log_int(50, 1000 if not replay else 300),
                "dtype": "float64" if replay else "float32", "replay": replay,
                "delay": rng.randrange(0, 12) if replay else 0, "steps": 300}
    if kind == "hines":
        return {"kind": kind, "neurons": log_int(20, 1024), "comps": log_int(220, 1000),
                "channels": rng.choice(("float32", "float64")), "steps": 200}
    return {"kind": kind, "rows": log_int(1000, 1_000_000)}


# ---- building -----------------------------------------------------------------------------------
_stream = None


def _program_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


class _Device:
    """A device array of the library as torch sees it; a tensor made from it keeps the network,
    which owns the memory, alive."""

    def __init__(self, net, ptr, n, dtype):
        self.net = net
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": np.dtype(dtype).str,
                                         "data": (int(ptr), False), "version": 3}


def _cuba_input(case, seed):
    """Potentials and connectivity of a CUBA network: v, (i, j) of the excitatory and of the
    inhibitory synapses."""
    n = case["n"]
    rng = np.random.default_rng([11, seed])
    v = rng.uniform(-60e-3, -50e-3, n)
    i, j = models.bernoulli_pairs(rng, n, n, min(1.0, CUBA_INDEGREE / n))
    exc = i < int(0.8 * n)
    return v, (i[exc], j[exc]), (i[~exc], j[~exc])


CUBA_WE, CUBA_WI = 1.62e-3, -9e-3     # V (examples/cuba.py:135-136)
CUBA = dict(El=-49e-3, taum=20e-3, taue=5e-3, taui=10e-3, ke=1.0, ki=1.0, Vt=-50e-3, Vr=-60e-3,
            refractory=5e-3, unless_refractory=True)


def _prepare_cuba(case, seed):
    net = Network(DT, seed=seed, stream=_program_stream().cuda_stream, small=case["small"])
    P = net.lif_group(case["n"], LIF(**CUBA), case["dtype"])
    v, exc, inh = _cuba_input(case, seed)
    net.set_state(P, "v", v)
    net.synapses(P, P, "ge", *exc, w_scalar=CUBA_WE)
    net.synapses(P, P, "gi", *inh, w_scalar=CUBA_WI)
    net.spike_monitor(P, MON)
    return _ready(net, [P], LIF_VARS, case["dtype"])


def _prepare_cuba_delays(case, seed):
    n = case["n"]
    rng = np.random.default_rng([12, seed])
    net = Network(DT, seed=seed, stream=_program_stream().cuda_stream)
    P = net.lif_group(n, LIF(**CUBA), case["dtype"])
    net.set_state(P, "v", rng.uniform(-60e-3, -50e-3, n))
    ne, p = int(0.8 * n), CUBA_INDEGREE / n
    net.synapses_random(P, P, "ge", p, 1, 20, CUBA_WE, seed, pre_range=(0, ne))
    net.synapses_random(P, P, "gi", p, 1, 20, CUBA_WI, seed + 7, pre_range=(ne, n))
    net.spike_monitor(P, MON)
    return _ready(net, [P], LIF_VARS, case["dtype"])


def _prepare_cobahh(case, seed):
    net = Network(DT, seed=seed, stream=_program_stream().cuda_stream,
                  one_launch=case["one_launch"])
    ids = models.build_cobahh(net, n=case["n"], p=P_CONNECT, dmin=DELAYS[0], dmax=DELAYS[1],
                              dtype=case["dtype"], seed_offset=seed, monitor_capacity=MON)
    return _ready(net, [ids["P"]], HH_VARS, case["dtype"])


def _prepare_batched(case, seed):
    net = Network(DT, seed=seed, stream=_program_stream().cuda_stream)
    sizes, _ = models.batch_sizes(case["instances"])
    we = np.random.default_rng([17, seed]).uniform(4e-9, 8e-9, len(sizes))
    ids = models.build_cobahh_batch(net, sizes, we, p=P_CONNECT, dmin=DELAYS[0],
                                    dmax=DELAYS[1], seed_offset=seed % 1_000_000,
                                    monitor_capacity=MON // len(sizes))
    return _ready(net, ids["groups"], HH_VARS, "float32")


def _prepare_propagation(case, seed):
    n_in, n_out = case["n_in"], case["n_out"]
    net = Network(DT, seed=seed, stream=_program_stream().cuda_stream)
    S = net.poisson_group(n_in, case["rate"], "float32")
    P = net.hh_group(n_out, models.cobahh_hh(), "float32")
    models.cobahh_init(net, P, n_out, np.random.default_rng([13, seed]))
    ne = int(0.8 * n_in)
    net.synapses_random(S, P, "ge", P_CONNECT, *DELAYS, 6e-9, seed, pre_range=(0, ne))
    net.synapses_random(S, P, "gi", P_CONNECT, *DELAYS, 67e-9, seed + 7, pre_range=(ne, n_in))
    net.spike_monitor(P, MON)
    # every slot of the delay ring holds spikes from the checkpoint on
    return _ready(net, [P], HH_VARS, "float32", fill=2 * DELAYS[1])


STDP_W = 0.01                    # largest weight (examples/stdp.py:125-186)


def _stdp_input(case, seed):
    """Initial weights, and the recorded spike trains (neuron, step) of a replayed input."""
    n_in, n_out = case["n_in"], case["n_out"]
    rng = np.random.default_rng([14, seed])
    w = rng.random(n_in * n_out) * STDP_W
    who = when = None
    if case["replay"]:
        hit = rng.random((case["steps"], n_in)) < 15.0 * DT * (10_000 / n_in) ** 0.5
        when, who = np.nonzero(hit)
    return w, who, when


def _prepare_stdp(case, seed):
    n_in, n_out, dtype = case["n_in"], case["n_out"], case["dtype"]
    net = Network(DT, seed=seed, stream=_program_stream().cuda_stream)
    w, who, when = _stdp_input(case, seed)
    if case["replay"]:
        inp = net.spikegen_group(n_in, who, when)
    else:
        inp = net.poisson_group(n_in, 15.0, dtype)
    out = net.lif_group(n_out, models.stdp_lif(), dtype)
    net.set_state(out, "v", -60e-3)
    i = np.repeat(np.arange(n_in, dtype=np.int32), n_out)
    j = np.tile(np.arange(n_out, dtype=np.int32), n_in)
    S = net.synapses(inp, out, "ge", i, j, w=w, delay=case["delay"],
                     stdp=models.stdp_rule(STDP_W))
    net.spike_monitor(out, MON)
    state = _ready(net, [out], ("v", "ge"), dtype)
    state["weights"] = S
    return state


def _ready(net, groups, variables, dtype, fill=0):
    """Finalizes the network, simulates `fill` steps and takes the checkpoint of every pass."""
    net.finalize()
    if fill:
        net.run(fill)
    net.store(0)
    views = {v: [torch.as_tensor(_Device(net, net.state_ptr(g, v), net.group_size(g), dtype),
                                 device="cuda") for g in groups] for v in variables}
    return {"net": net, "views": views}


def _morphologies(case, seed):
    """Trees of sections (the same for every seed), their geometry and the soma currents."""
    m = models.random_morphologies(case["neurons"], np.random.default_rng(15),
                                   comp_range=(200, case["comps"]))
    rng = np.random.default_rng([15, seed])
    m["diameter"] = rng.uniform(0.5e-6, 2e-6, len(m["diameter"]))
    m["length"] = rng.uniform(5e-6, 50e-6, len(m["length"]))
    return m, rng.uniform(0.2e-9, 1e-9, size=case["neurons"])


def _prepare_hines(case, seed):
    net = Network(HINES_DT, seed=seed, stream=_program_stream().cuda_stream)
    m, current = _morphologies(case, seed)
    hb = net.hines_batch(m["comp_off"], m["sec_off"], m["sec_start"], m["sec_end"],
                         m["sec_parent"], m["diameter"], m["length"],
                         HinesParams(channel_dtype=case["channels"]))
    for var, x in models.hines_rest_state().items():
        hb.set_state(var, x)
    hb.set_current(current)
    return {"net": net, "batch": hb}


def _surrogate_input(case, seed):
    """States (v, m, h, n) of neurons, the gates one step later, and the network's parameters
    and scaling."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["rows"]
    x = torch.rand((n, 4), device="cuda", generator=g)
    t = torch.clamp(x[:, 1:] + 0.01 * torch.randn((n, 3), device="cuda", generator=g), 0, 1)
    x[:, 0] = x[:, 0] * 0.13 - 0.085
    rng = np.random.default_rng([16, seed])
    params = np.concatenate([
        (rng.uniform(-1, 1, (fan_out, fan_in)) * math.sqrt(6 / (fan_in + fan_out))).ravel()
        if fan_in else 0.1 * rng.standard_normal(fan_out)
        for fan_out, fan_in in ((64, 4), (64, 0), (64, 64), (64, 0), (3, 64), (3, 0))])
    scaling = np.array([-0.02, 0.5, 0.5, 0.5, 1 / 0.065, 2, 2, 2, 0.01, 0.01, 0.01])
    return x, t, params.astype(np.float32), scaling.astype(np.float32)


def _prepare_surrogate(case, seed):
    x, t, params, scaling = _surrogate_input(case, seed)
    torch.cuda.synchronize()
    net = GatingSurrogate(seed=1, stream=_program_stream().cuda_stream)
    net.params = params
    net.scaling = scaling
    return {"mlp": net, "x": x, "t": t}


_PREPARE = {"cuba": _prepare_cuba, "cuba_delays": _prepare_cuba_delays,
            "cobahh": _prepare_cobahh, "batched": _prepare_batched,
            "propagation": _prepare_propagation, "stdp": _prepare_stdp,
            "hines": _prepare_hines, "surrogate": _prepare_surrogate}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["steps"] = case.get("steps")
    return state


# ---- one pass -----------------------------------------------------------------------------------
def run(state):
    if "mlp" in state:
        with torch.cuda.stream(_program_stream()):
            y = state["mlp"].forward(state["x"])
            grad, loss = state["mlp"].grad(state["x"], state["t"])
        return {"gates": y, "grad": grad, "loss": loss}
    if "batch" in state:
        hb = state["batch"]
        hb.run(state["steps"])      # the batch runs on from where its last run ended
        return {**{v: hb.get_state(v) for v in ("v", "m", "h", "n")},
                "spikes": hb.spike_counts()}
    net = state["net"]
    net.restore(0)
    net.run(state["steps"])
    with torch.cuda.stream(_program_stream()):
        out = {v: x[0] if len(x) == 1 else torch.cat(x) for v, x in state["views"].items()}
    if "weights" in state:
        out["w"] = net.syn_get(state["weights"], "w")
    return out


# ---- the least a pass can do --------------------------------------------------------------------
# Operations of one neuron's step: the exponential-Euler update of COBAHH (9 exponentials, 7
# quotients, the sums and products around them), the exact LIF update.
HH_FLOPS, LIF_FLOPS = 250, 12
L2_BYTES = 126e6


def _network_work(n, state_bytes, flops, steps, events, event_bytes):
    """State in and out once per pass, or once per step where it does not fit the L2 cache, and
    per synaptic event the target index (and what the event updates besides it)."""
    moves = steps if n * state_bytes / 2 > L2_BYTES else 1
    return {"bytes": moves * n * state_bytes + events * event_bytes,
            "flops": steps * n * flops + events}


def work(case):
    kind, k = case["kind"], case.get("steps")
    if kind in ("cuba", "cuba_delays"):
        r = 8 if case["dtype"] == "float64" else 4
        n = case["n"]
        events = 5.0 * n * k * DT * CUBA_INDEGREE            # ~5 Hz
        return _network_work(n, 8 * r, LIF_FLOPS, k, events, 4)
    if kind == "cobahh":
        r = 8 if case["dtype"] == "float64" else 4
        n = case["n"]
        events = 3.0 * n * k * DT * P_CONNECT * n             # ~3 Hz
        return _network_work(n, 14 * r, HH_FLOPS, k, events, 4)
    if kind == "batched":
        n = 15_340 * case["instances"]     # mean of the log-uniform sizes on [1e3, 6.4e4]
        # mean square of the sizes; ~3 Hz
        events = 3.0 * k * DT * P_CONNECT * 4.92e8 * case["instances"]
        return _network_work(n, 56, HH_FLOPS, k, events, 4)
    if kind == "propagation":
        events = case["rate"] * case["n_in"] * k * DT * P_CONNECT * case["n_out"]
        return _network_work(case["n_out"], 56, HH_FLOPS, k, events, 4)
    if kind == "stdp":
        # every output spike (about every tenth step, every second under the configured
        # drive) updates the weights of all inputs; the weights are read out once
        r = 8 if case["dtype"] == "float64" else 4
        n_syn = case["n_in"] * case["n_out"]
        events = n_syn * k * (0.1 if case["replay"] else 0.4 * case["n_in"] / 10_000)
        return {"bytes": 2 * r * n_syn, "flops": 4 * events}
    if kind == "hines":
        comps = case["neurons"] * (200 + case["comps"]) / 2
        r = 8 if case["channels"] == "float64" else 4
        return {"bytes": comps * 2 * (8 + 3 * r), "flops": 200 * comps * k}
    # forward 2 (4 64 + 64 64 + 64 3) operations per row; the gradient's pass again and twice
    # that backward
    return {"bytes": case["rows"] * (16 + 12 + 12), "flops": case["rows"] * 9088 * 4}


# ---- 64-bit values ------------------------------------------------------------------------------
def exact(case, seed):
    """COBAHH-shaped networks have none: their connectivity is generated by the library, and a
    window holds thousands of spikes whose times follow every rounding of the coupled
    equations.  The same for inputs drawn by the library (the Poisson-driven STDP network) and
    the delayed CUBA networks.  A large batch of morphologies would take minutes."""
    kind = case["kind"]
    if kind == "cuba" and case["dtype"] == "float64":
        return _exact_cuba(case, seed)
    if kind == "stdp" and case["replay"]:
        return _exact_stdp(case, seed)
    if kind == "hines" and case["channels"] == "float64" and case["neurons"] <= 128:
        return _exact_hines(case, seed)
    if kind == "surrogate":
        return _exact_surrogate(case, seed)
    return None


def _steps_past(t, dt=DT):
    return np.floor((t + 1e-3 * dt) / dt)


def _exact_cuba(case, seed):
    n = case["n"]
    v, exc, inh = _cuba_input(case, seed)
    taum, taue, taui, El = CUBA["taum"], CUBA["taue"], CUBA["taui"], CUBA["El"]
    A, De, Di = (math.exp(-DT / tau) for tau in (taum, taue, taui))
    Be, Bi = taue / (taue - taum) * (De - A), taui / (taui - taum) * (Di - A)

    def rows(i, j):
        return np.searchsorted(i, np.arange(n + 1)), j

    oe, je = rows(*exc)
    oi, ji = rows(*inh)
    ge, gi, last = np.zeros(n), np.zeros(n), np.full(n, -1e4)
    hold = _steps_past(CUBA["refractory"])
    for ts in range(case["steps"]):
        t = ts * DT
        ready = _steps_past(t - last) >= hold
        v = np.where(ready, El + A * (v - El) + Be * ge + Bi * gi, v)
        ge, gi = De * ge, Di * gi
        spikes = np.nonzero((v > CUBA["Vt"]) & ready)[0]
        for off, post, g, w in ((oe, je, ge, CUBA_WE), (oi, ji, gi, CUBA_WI)):
            for s in spikes:
                g[post[off[s]:off[s + 1]]] += w      # a bundle's targets are distinct
        last[spikes] = t
        v[spikes] = CUBA["Vr"]
    return {"v": v, "ge": ge, "gi": gi, "lastspike": last}


def _exact_stdp(case, seed):
    n_in, n_out = case["n_in"], case["n_out"]
    w, who, when = _stdp_input(case, seed)
    w = w.reshape(n_in, n_out)
    lif, rule = models.stdp_lif(), models.stdp_rule(STDP_W)
    A, De = math.exp(-DT / lif.taum), math.exp(-DT / lif.taue)
    Be = lif.ke * lif.taue / (lif.taue - lif.taum) * (De - A)
    dpre, dpost = math.exp(-DT / rule.taupre), math.exp(-DT / rule.taupost)
    v, ge = np.full(n_out, -60e-3), np.zeros(n_out)
    apre, apost = np.zeros(n_in), np.zeros(n_out)   # every synapse's traces, per neuron
    for ts in range(case["steps"]):
        v = lif.El + A * (v - lif.El) + Be * ge
        ge = De * ge
        apre, apost = dpre * apre, dpost * apost
        spikes = np.nonzero(v > lif.Vt)[0]
        arrive = who[when == ts - case["delay"]]
        ge += w[arrive].sum(axis=0)
        apre[arrive] += rule.dApre
        w[arrive] = np.clip(w[arrive] + apost, rule.wmin, rule.wmax)
        apost[spikes] += rule.dApost
        w[:, spikes] = np.clip(w[:, spikes] + apre[:, None], rule.wmin, rule.wmax)
        v[spikes] = lif.Vr
    return {"v": v, "ge": ge, "w": w.ravel()}


def _exact_hines(case, seed):
    """Backward Euler of the cable equation on the tree of compartments and section nodes
    (Kirchhoff's law at each node), eliminated towards the root, all neurons side by side."""
    m, current = _morphologies(case, seed)
    p = HinesParams()
    nb = case["neurons"]
    d, L = m["diameter"], m["length"]
    area, rl = math.pi * d * L, math.pi * d * d / (2 * L)
    size = int(np.max(np.diff(m["comp_off"]) + np.diff(m["sec_off"])))
    # per neuron a list of unknowns (compartments, and after each section its end node), a
    # parent before its children; the coupling to the parent in either equation
    parent = np.zeros((size, nb), np.int64)
    diag = np.ones((size, nb))
    down, up = np.zeros((size, nb)), np.zeros((size, nb))   # own equation, parent's equation
    place, is_comp = np.zeros(len(d), np.int64), np.zeros((size, nb), bool)
    for b in range(nb):
        c0, s0 = m["comp_off"][b], m["sec_off"][b]
        node, k = {}, 0

        def couple(child, par, g, child_area, par_area):
            parent[child, b] = par
            down[child, b], up[child, b] = g / child_area, g / par_area
            diag[child, b] -= g / child_area
            diag[par, b] -= g / par_area

        for s in range(m["sec_off"][b + 1] - s0):
            first = True
            for c in range(c0 + m["sec_start"][s0 + s], c0 + m["sec_end"][s0 + s]):
                place[c], is_comp[k, b] = k, True
                diag[k, b] = -p.Cm / HINES_DT
                if not first:
                    couple(k, k - 1, 1 / (p.Ri * (1 / rl[c - 1] + 1 / rl[c])), area[c],
                           area[c - 1])
                elif s > 0:
                    couple(k, node[m["sec_parent"][s0 + s]], rl[c] / p.Ri, area[c], 1.0)
                first, k = False, k + 1
            diag[k, b] = 0.0
            couple(k, k - 1, rl[c] / p.Ri, 1.0, area[c])
            node[s], k = k, k + 1
    cols = np.arange(nb)
    rest = models.hines_rest_state()
    v = np.full((size, nb), rest["v"])
    x = {g: np.full((size, nb), rest[g]) for g in "mhn"}
    above, spikes = np.zeros(nb, bool), np.zeros(nb, np.int64)
    soma = current / area[m["comp_off"][:-1]]

    def over_expm1(z):
        return np.where(np.abs(z) < 1e-16, 1.0, z / np.expm1(np.where(z == 0, 1.0, z)))

    for _ in range(case["steps"]):
        gna, gk = p.gNa * x["m"] ** 3 * x["h"], p.gK * x["n"] ** 4
        dg = np.where(is_comp, diag - (p.gl + gna + gk), diag)
        I0 = p.gl * p.El + gna * p.ENa + gk * p.EK
        I0[0] += soma
        rhs = np.where(is_comp, -p.Cm / HINES_DT * v - I0, 0.0)
        rates = {"m": (1000 * over_expm1((25e-3 - v) / 10e-3), 4000 * np.exp(-v / 18e-3)),
                 "h": (70 * np.exp(-v / 20e-3), 1000 / (np.exp((30e-3 - v) / 10e-3) + 1)),
                 "n": (100 * over_expm1((10e-3 - v) / 10e-3), 125 * np.exp(-v / 80e-3))}
        for g, (a, b) in rates.items():
            x[g] = a / (a + b) + (x[g] - a / (a + b)) * np.exp(-(a + b) * HINES_DT)
        for k in range(size - 1, 0, -1):
            f = up[k] / dg[k]
            dg[parent[k], cols] -= f * down[k]
            rhs[parent[k], cols] -= f * rhs[k]
        v = np.empty_like(rhs)
        v[0] = rhs[0] / dg[0]
        for k in range(1, size):
            v[k] = (rhs[k] - down[k] * v[parent[k], cols]) / dg[k]
        now = v[0] > p.Vthr
        spikes += now & ~above
        above = now
    b_of = np.repeat(cols, np.diff(m["comp_off"]))
    return {"v": v[place, b_of], **{g: x[g][place, b_of] for g in "mhn"}, "spikes": None}


def _exact_surrogate(case, seed):
    x, t, params, scaling = _surrogate_input(case, seed)
    q = torch.from_numpy(params.astype(np.float64)).cuda().requires_grad_()
    sc = torch.from_numpy(scaling.astype(np.float64)).cuda()
    W1, b1, W2, b2, W3, b3 = (
        a.reshape(s) for a, s in zip(torch.split(q, [256, 64, 4096, 64, 192, 3]),
                                     ((64, 4), (64,), (64, 64), (64,), (3, 64), (3,))))
    n, gates, loss = case["rows"], [], 0.0
    for lo in range(0, n, 1 << 17):
        xd, td = x[lo:lo + (1 << 17)].double(), t[lo:lo + (1 << 17)].double()
        h = torch.tanh(((xd - sc[:4]) * sc[4:8]) @ W1.T + b1)
        y = torch.tanh(h @ W2.T + b2) @ W3.T + b3
        gates.append(torch.clamp(xd[:, 1:] + sc[8:] * y.detach(), 0, 1))
        part = ((y - (td - xd[:, 1:]) / sc[8:]) ** 2).sum() / n
        part.backward(retain_graph=True)
        loss += part.item()
    return {"gates": torch.cat(gates), "grad": q.grad.cpu().numpy(), "loss": loss}
