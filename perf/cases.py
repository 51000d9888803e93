"""Workloads that the framework is timed on, through its public entry points.

What a user has the framework do, over the sizes it is used at:

* a simulation from its start (no synapses yet: the stated 2,000-, 1M- and
  4M-neuron runs and the batched ensembles spend their time here);
* a simulation resumed from a mature network, with synapses in both signs and
  calcium around its set point, so that activity is coupled through spikes and
  every plasticity update commits, deletes, searches and connects;
* a block of activity steps alone (the NeuronModel plugin's half), with the
  other neuron models;
* the Algorithm plugin's half alone: an octree update and a Barnes-Hut search
  for every vacant axon, dense and sparse, with each probability kernel;
* the serving loop over a handful of requests of uneven size.

Small cases return the whole state; from 200,000 neurons on a simulation
returns what a monitor reads of it (calcium and spike flags through the pinned
snapshot), since such a run does not copy every array out between its parts.
"""
import math

import numpy as np
import torch

import relearn_b200 as R
from relearn_b200 import workloads
from relearn_b200.serving import Server

DENSITY = 1000.0  # cubic micrometres per neuron, as in every stated configuration
BETA = 0.0065     # calcium per spike that holds a mature network at its target


def listed():
    return [
        # the smallest stated network, resumed with synapses: launch latency
        {"name": "resume_2k_f64", "kind": "sim", "n": 2000, "precision": 0, "model": 0, "placement": "uniform", "edges": 4.0, "steps": 500, "tune": 0},
        # the size of the reference's positions file (odd), clustered
        {"name": "resume_52k_f64", "kind": "sim", "n": 51842, "precision": 0, "model": 0, "placement": "mixture", "edges": 3.0, "steps": 300, "tune": 0},
        # the headline run: 1M neurons from the start, FP64 drop-in
        {"name": "start_1m_f64", "kind": "sim", "n": 1000000, "precision": 0, "model": 0, "placement": "uniform", "edges": 0.0, "steps": 500, "tune": 1},
        # 1M neurons once synapses exist, both precision forms
        {"name": "resume_1m_f64", "kind": "sim", "n": 1000000, "precision": 0, "model": 0, "placement": "uniform", "edges": 2.0, "steps": 300, "tune": 1},
        {"name": "resume_1m_f32", "kind": "sim", "n": 1000000, "precision": 1, "model": 0, "placement": "mixture", "edges": 4.0, "steps": 300, "tune": 1},
        # the precision form's stated size
        {"name": "start_4m_f32", "kind": "sim", "n": 4000000, "precision": 1, "model": 0, "placement": "uniform", "edges": 0.0, "steps": 300, "tune": 0},
        # the batched form: networks of log-uniform size in one context
        {"name": "ensemble_48_f32", "kind": "ensemble", "networks": 48, "low": 5000, "high": 250000, "precision": 1, "steps": 500, "spread": 7},
        # the NeuronModel plugin alone, another model, a ragged size
        {"name": "activity_aeif_100k_f64", "kind": "activity", "n": 100003, "precision": 0, "model": 3, "placement": "uniform", "edges": 5.0, "steps": 100},
        # the Algorithm plugin alone: every neuron searches (the reference's own search benchmark)
        {"name": "search_dense_1m_f64", "kind": "search", "n": 1000000, "precision": 0, "kernel": 0, "placement": "uniform", "share": 1.0, "theta": 0.3, "tune": 0},
        # a growing network: one neuron in fifty has a vacant axon
        {"name": "search_sparse_1m_f64", "kind": "search", "n": 1000000, "precision": 0, "kernel": 0, "placement": "uniform", "share": 0.02, "theta": 0.3, "tune": 1},
        # the FP32 form on a clustered, ragged network
        {"name": "search_dense_300k_f32", "kind": "search", "n": 300007, "precision": 1, "kernel": 0, "placement": "mixture", "share": 1.0, "theta": 0.3, "tune": 0},
        # a sweep served: eight requests of uneven size submitted together
        {"name": "serve_8_f32", "kind": "serve", "requests": 8, "low": 2000, "high": 300000, "precision": 1, "steps": 1000, "spread": 3},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the same ranges: 1,000 to 1.2M neurons, ragged sizes,
    both precision forms, every neuron model and probability kernel."""
    kind = rng.choice(["sim", "sim", "sim", "activity", "search", "search", "ensemble", "serve"])
    precision = rng.choice([0, 1])
    placement = rng.choice(["uniform", "mixture"])
    if kind == "sim":
        n = _log(rng, 1000, 1200000)
        steps = max(100, min(500, int(2e8 / n) // 100 * 100))
        return {"kind": kind, "n": n, "precision": precision, "model": 0, "placement": placement,
                "edges": rng.choice([0.0, round(rng.uniform(1.0, 6.0), 2), round(rng.uniform(1.0, 6.0), 2)]), "steps": steps, "tune": rng.choice([0, 1])}
    if kind == "activity":
        n = _log(rng, 1000, 1000000)
        return {"kind": kind, "n": n, "precision": precision, "model": rng.choice([0, 1, 2, 3]), "placement": placement,
                "edges": rng.choice([0.0, round(rng.uniform(1.0, 6.0), 2)]), "steps": rng.choice([37, 100, 150])}
    if kind == "search":
        n = _log(rng, 2000, 800000)
        return {"kind": kind, "n": n, "precision": precision, "kernel": rng.choice([0, 0, 0, 1, 2, 3]), "placement": placement,
                "share": rng.choice([1.0, round(math.exp(rng.uniform(math.log(2e-3), 0.0)), 4)]), "theta": rng.choice([0.2, 0.3, 0.5]), "tune": rng.choice([0, 1])}
    if kind == "ensemble":
        return {"kind": kind, "networks": rng.randint(3, 40), "low": 5000, "high": _log(rng, 20000, 250000), "precision": precision, "steps": rng.choice([100, 300, 500]),
                "spread": rng.randint(1, 10**6)}
    return {"kind": kind, "requests": rng.randint(3, 8), "low": 2000, "high": _log(rng, 20000, 250000), "precision": precision, "steps": rng.choice([300, 700, 1000]),
            "spread": rng.randint(1, 10**6)}


# ------------------------------------------------------------------- inputs
def _side(n):
    return (DENSITY * n) ** (1.0 / 3.0)


def _place(n, placement, seed):
    side = _side(n)
    if placement == "uniform":
        return workloads.uniform_cube(n, side, seed)
    # a cluster's width scales with the cube, as 200 um does in the 10,000 um cube
    return workloads.gaussian_mixture(n, side, seed, components=64, std=0.02 * side)


def _params(case, n, seed):
    p = R.default_params(n, _side(n))
    p["seed"] = seed * 1000003 + 17
    p["precision"] = case["precision"]
    p["neuron_model"] = case.get("model", 0)
    p["theta"] = case.get("theta", 0.3)
    kernel = case.get("kernel", 0)
    p["kernel_type"] = kernel
    if kernel == 1:
        p["kernel_k"], p["kernel_scale"] = 2.0, 375.0
    elif kernel == 2:
        p["linear_cutoff"] = 2000.0
    elif kernel == 3:
        p["kernel_k"], p["kernel_scale"] = 2.0, 1.0 / 750.0**2
    if case.get("model", 0) == 1:  # the Poisson model's input is a small drive towards its threshold
        p["noise_mean"], p["noise_stddev"], p["conductance"] = 0.0, 0.1, 0.3
    elif case.get("model", 0) == 2:  # FitzHugh-Nagumo fires on a current of about one
        p["noise_mean"], p["noise_stddev"], p["conductance"] = 0.7, 0.5, 0.3
    elif case.get("model", 0) == 3:  # AEIF: picoamperes
        p["noise_mean"], p["noise_stddev"], p["conductance"] = 600.0, 200.0, 300.0
    if case.get("edges", 0.0) > 0.0:
        p["beta"] = BETA
    return p


def _edges(n, per_neuron, sig, rng):
    m = int(n * per_neuron)
    s = rng.integers(0, n, m)
    t = (s + rng.integers(1, n, m)) % n
    w = np.where(sig[s] == 0, 1, -1).astype(np.int32)
    return t.astype(np.uint32), s.astype(np.uint32), w


def _initial(case, seed):
    """Everything the simulation and activity cases start from."""
    n = case["n"]
    rng = np.random.default_rng([seed, n, 5])
    params = _params(case, n, seed)
    pos = _place(n, case["placement"], seed)
    sig = workloads.signal_types(n, seed)
    d = {"params": params, "pos": pos, "sig": sig}
    if case.get("edges", 0.0) > 0.0:
        d["edges"] = _edges(n, case["edges"], sig, rng)
        d["calcium"] = np.clip(params["target_calcium"] + 0.03 * rng.standard_normal(n), 0.0, None)
        if case["model"] == 0:
            d["x"] = rng.uniform(-70.0, -55.0, n)
            d["u"] = 0.2 * d["x"]
        d["fraction"] = [rng.random(n) for _ in range(3)]
        d["free"] = [np.zeros(n, np.uint32), (rng.random(n) < 0.05).astype(np.uint32), (rng.random(n) < 0.05).astype(np.uint32)]
    return d


def _network(case, d):
    net = R.Network(d["params"])
    net.set_positions(d["pos"], d["sig"])
    if "edges" in d:
        t, s, w = d["edges"]
        net.load_network(t, s, w)
        for k in range(3):
            e = net.get_elements(k)
            net.set_elements(k, e["grown"] + d["fraction"][k] + d["free"][k], e["delta"], e["connected"], e["vacant"] + d["free"][k])
        net.set_neurons(x=d.get("x"), u=d.get("u"), calcium=d["calcium"])
    if case.get("tune", 0):
        net.autotune(1)
    return net


def _ensemble(case, seed):
    rng = np.random.default_rng(case["spread"])
    nets, pos, sig = [], [], []
    for k in range(case["networks"]):
        n = int(np.exp(rng.uniform(np.log(case["low"]), np.log(case["high"]))))
        nets.append(dict(num_neurons=n, seed=seed * 100003 + k, side=_side(n), theta=float(rng.choice([0.2, 0.3, 0.5])),
                         sigma=float(rng.choice([500.0, 750.0, 1000.0])), growth_rate=float(np.exp(rng.uniform(np.log(1e-5), np.log(1e-3))))))
        pos.append(workloads.uniform_cube(n, nets[-1]["side"], seed * 1009 + k))
        sig.append(workloads.signal_types(n, seed * 1009 + k))
    return nets, np.concatenate(pos), np.concatenate(sig)


def _requests(case, seed):
    rng = np.random.default_rng(case["spread"])
    out = []
    for k in range(case["requests"]):
        n = int(np.exp(rng.uniform(np.log(case["low"]), np.log(case["high"]))))
        net = dict(num_neurons=n, seed=seed * 1000003 + k, side=_side(n), theta=float(rng.uniform(0.2, 0.5)), sigma=750.0,
                   growth_rate=float(np.exp(rng.uniform(np.log(1e-5), np.log(1e-3)))))
        out.append((net, *workloads.request_inputs(net)))
    return out


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy(), torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sim", "activity"):
        net = _network(case, _initial(case, seed))
        st = {"kind": kind, "net": net, "step": 1, "steps": case["steps"], "whole": kind == "activity" or case["n"] < 200000,
              "counters": case["precision"] == 0, "room": int(case["n"] * (case["edges"] + 1.0))}
        if not st["whole"]:
            st["calcium"], st["fired"] = _pinned(case["n"])
        return st
    if kind == "ensemble":
        nets, pos, sig = _ensemble(case, seed)
        base = R.default_params(1, 1.0)
        base["precision"] = case["precision"]
        net = R.Network(base, networks=nets)
        net.set_positions(pos, sig)
        calcium, fired = _pinned(len(sig))
        return {"kind": "sim", "net": net, "step": 1, "steps": case["steps"], "whole": False, "counters": False, "calcium": calcium, "fired": fired}
    if kind == "search":
        n = case["n"]
        net = R.Network(_params(case, n, seed))
        sig = workloads.signal_types(n, seed)
        net.set_positions(_place(n, case["placement"], seed), sig)
        if case["tune"]:
            net.autotune(1)
        rng = np.random.default_rng([seed, n, 9])
        axons = np.zeros(n, np.uint32)
        axons[rng.permutation(n)[:max(1, round(n * case["share"]))]] = 1
        one = np.ones(n, np.uint32)
        return {"kind": kind, "net": net, "step": 1, "axons": axons, "exc": one, "inh": one}
    base = R.default_params(1, 1.0)
    base["precision"] = case["precision"]
    return {"kind": kind, "server": Server(base, hbm_budget_bytes=20e9, slots=8), "requests": _requests(case, seed), "steps": case["steps"]}


# ----------------------------------------------------------------- one pass
def _state(st):
    net = st["net"]
    out = dict(net.neurons())
    for k, name in enumerate(("axons", "dendrites_exc", "dendrites_inh")):
        out[name] = net.get_elements(k)
    edges = net.edges()
    room = max(st["room"], len(edges[0]))  # the list at a fixed length, as a recorder of several times keeps it
    out["edges"] = {}
    for name, e in zip(("target", "source", "weight"), edges):
        out["edges"][name] = np.zeros(room, e.dtype)
        out["edges"][name][:len(e)] = e
    return out


def run(st):
    if st["kind"] == "search":
        net = st["net"]
        net.prepare_update_connectivity(st["axons"], st["exc"], st["inh"])
        req = net.find_targets(st["step"])
        st["step"] += 1
        return {k: req[k] for k in ("target", "source", "j", "signal")}
    if st["kind"] == "serve":
        srv = st["server"]
        ids = [srv.submit(net, pos, sig, st["steps"], keep_state=True) for net, pos, sig in st["requests"]]
        done = {}
        while len(done) < len(ids):
            done.update((d["id"], d) for d in srv.poll(wait_ms=200))
        return [srv.fetch(done[i]) for i in ids]
    net = st["net"]
    if st["kind"] == "activity":
        net.activity_block(st["step"], st["steps"])
    else:
        net.simulate(st["step"], st["steps"])
    st["step"] += st["steps"]
    if st["whole"]:
        return _state(st)
    net.snapshot_neurons(st["calcium"], st["fired"])
    net.snapshot_wait()
    out = {"calcium": st["calcium"], "fired": st["fired"]}
    if st["counters"]:
        s = net.stats()
        out["counters"] = np.array([s["searches"], s["synapses_created"], s["synapses_deleted"], s["bound_to_delete"]])
    return out


# -------------------------------------------------------------------- floors
def _count(case):
    if case["kind"] == "ensemble":
        rng = np.random.default_rng(case["spread"])
        total = 0
        for _ in range(case["networks"]):
            total += int(np.exp(rng.uniform(np.log(case["low"]), np.log(case["high"]))))
            rng.choice(3), rng.choice(3), rng.uniform()
        return total
    if case["kind"] == "serve":
        rng = np.random.default_rng(case["spread"])
        total = 0
        for _ in range(case["requests"]):
            total += int(np.exp(rng.uniform(np.log(case["low"]), np.log(case["high"]))))
            rng.uniform(), rng.uniform()
        return total
    return case["n"]


def work(case):
    """Bytes: the state once in and once out, and the synapse list (or the
    search's octree records and requests).  Operations: the model's h = 10
    substeps, calcium, three growth curves and one normal draw per
    neuron-step; a distance, an acceptance test and a weight per node that a
    search has to visit (about 185 log2 n at theta = 0.3)."""
    n = _count(case)
    wide = 8 if case["precision"] == 0 else 4
    if case["kind"] == "search":
        searches = n * case["share"]
        nodes = 185.0 * math.log2(n) * (0.3 / case["theta"]) ** 2
        return {"bytes": 1.48 * n * (32 if wide == 8 else 16) + 12.0 * n + 16.0 * searches, "flops": searches * nodes * 40.0}
    per_step = {0: 310.0, 1: 150.0, 2: 330.0, 3: 600.0}[case.get("model", 0)]
    state = 2 * (8.0 + 6 * wide + 1)
    return {"bytes": n * state + 12.0 * n * case.get("edges", 0.0), "flops": n * case["steps"] * per_step}


def tolerance(case):
    if case["precision"] == 0:
        return "exact"  # the FP64 form promises the reference's bits and its connectome
    if case["kind"] == "search":
        return {"rel": 0.0, "differ": 2e-3}  # picks within rounding of a boundary of the running sum
    # single precision moves a few spikes by a step, and those neurons' state with them
    return {"rel": 5e-3, "max": 0.9, "differ": 5e-3}


# ---------------------------------------------------- the same in 64 bits
_M = 0xFFFFFFFF


def _philox(c, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    x, y, z, w = c
    for r in range(10):
        p0, p1 = x * 0xD2511F53, z * 0xCD9E8D57
        a = (k0 + r * 0x9E3779B9) & _M
        b = (k1 + r * 0xBB67AE85) & _M
        x, y, z, w = ((p1 >> 32) & _M) ^ y ^ a, p1 & _M, ((p0 >> 32) & _M) ^ w ^ b, p0 & _M
    return x, y, z, w


def _activity64(n, steps, p, nets, edges=None, x=None, u=None, calcium=None):
    """`steps` activity steps in plain 64-bit torch.  nets: (count, seed,
    growth rates) per network.  Returns x, u, calcium, the last input and the
    growth deltas."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    local = torch.cat([torch.arange(c, device=dev) for c, _, _ in nets])
    k0 = torch.cat([torch.full((c,), s & _M, device=dev) for c, s, _ in nets]) if len(nets) > 1 else nets[0][1] & _M
    k1 = torch.cat([torch.full((c,), s >> 32, device=dev) for c, s, _ in nets]) if len(nets) > 1 else nets[0][1] >> 32
    nu = torch.cat([torch.tensor(g, **f64).reshape(3, 1).expand(3, c) for c, _, g in nets], dim=1)
    model, h, hc = p["neuron_model"], p["h_model"], p["h_calcium"]
    rest = {0: p["iz_c"], 1: 0.0, 2: p["fhn_init_x"], 3: p["aeif_E_L"]}[model]
    x = torch.full((n,), float(rest), **f64) if x is None else torch.tensor(x, **f64)
    u = torch.full((n,), p["fhn_init_w"] if model == 2 else 0.0, **f64) if u is None else torch.tensor(u, **f64)
    ca = torch.full((n,), p["initial_calcium"], **f64) if calcium is None else torch.tensor(calcium, **f64)
    fired = torch.zeros(n, **f64)
    delta = torch.zeros(3, n, **f64)
    inp = torch.zeros(n, **f64)
    if edges is not None:
        tgt, src, wt = (torch.tensor(np.asarray(e, np.int64), device=dev) for e in edges)
        wt = wt.to(torch.float64)
    eta = torch.tensor(p["min_calcium"], **f64).reshape(3, 1)
    eps = torch.clamp(eta, min=p["target_calcium"])
    zero = torch.zeros_like(local)
    for k in range(steps):
        step = 1 + k
        words = _philox((zero + step, local >> 1, zero, zero + (3 << 24)), k0, k1)
        odd = (local & 1) == 1
        bits = (torch.where(odd, words[2], words[0]) << 21) | (torch.where(odd, words[3], words[1]) >> 11)
        z = torch.special.ndtri((bits.to(torch.float64) + 0.5) * 2.0**-53)
        inp = p["noise_mean"] + p["noise_stddev"] * z
        if edges is not None:
            inp = inp + p["conductance"] * torch.zeros(n, **f64).index_add_(0, tgt, wt * fired[src])
        spiked = torch.zeros(n, dtype=torch.bool, device=dev)
        if model == 1:
            for _ in range(h):
                x = x + ((p["poisson_x0"] - x) / p["poisson_tau_x"] + inp) / h
            q = _philox((zero + step, local, zero, zero + (5 << 24)), k0, k1)
            threshold = ((q[0] << 21) | (q[1] >> 11)).to(torch.float64) * 2.0**-53
            ready = u == 0.0
            spiked = ready & (x >= threshold)
            u = torch.where(spiked, torch.full_like(u, float(p["poisson_refractory"])), torch.where(ready, u, u - 1.0))
        elif model == 2:
            for _ in range(h):
                dx = x - x * x * x / 3.0 - u + inp
                dw = p["fhn_phi"] * (x + p["fhn_a"] - p["fhn_b"] * u)
                x, u = x + dx / h, u + dw / h
            spiked = (u > x - x * x * x / 3.0) & (x > 1.0)
        else:
            for _ in range(h):
                if model == 0:
                    dx = p["iz_k1"] * x * x + p["iz_k2"] * x + p["iz_k3"] - u + inp
                    du = p["iz_a"] * (p["iz_b"] * x - u)
                    top, reset, jump = p["iz_v_spike"], p["iz_c"], p["iz_d"]
                else:
                    g, e_l, d_t = p["aeif_g_L"], p["aeif_E_L"], p["aeif_d_T"]
                    dx = (-g * (x - e_l) + g * d_t * torch.exp((x - p["aeif_V_T"]) / d_t) - u + inp) / p["aeif_C"]
                    du = (p["aeif_a"] * (x - e_l) - u) / p["aeif_tau_w"]
                    top, reset, jump = p["aeif_V_spike"], e_l, p["aeif_b"]
                xn, un = x + dx / h, u + du / h
                hit = xn >= top
                xn = torch.where(hit, torch.full_like(xn, reset), xn)
                un = torch.where(hit, un + jump, un)
                x, u = torch.where(spiked, x, xn), torch.where(spiked, u, un)
                spiked = spiked | hit
        fired = spiked.to(torch.float64)
        for _ in range(hc):
            ca = ca + (ca * (-1.0 / p["tau_c"]) + p["beta"] * fired) / hc
        xi, zeta = (eta + eps) * 0.5, (eta - eps) / 1.6651092223153955
        curve = 2.0 * torch.exp(-(((ca - xi) / zeta) ** 2)) - 1.0
        flat = torch.where(ca == eta, torch.zeros_like(curve), torch.full_like(curve, -1.0))
        delta = delta + torch.where(eta == eps, flat, curve) * nu
    out = [v.cpu().numpy() for v in (x, u, ca, inp)]
    return out[0], out[1], out[2], out[3], delta.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    base = R.default_params(1, 1.0)
    if kind == "ensemble":
        nets, _, _ = _ensemble(case, seed)
        per = [(d["num_neurons"], d["seed"], (d["growth_rate"],) * 3) for d in nets]
        return {"calcium": _activity64(sum(c for c, _, _ in per), case["steps"], base, per)[2], "fired": None}
    if kind == "serve":
        out = []
        for net, _, _ in _requests(case, seed):
            n = net["num_neurons"]
            calcium = _activity64(n, case["steps"], base, [(n, net["seed"], (net["growth_rate"],) * 3)])[2]
            out.append({"x": None, "u": None, "calcium": calcium, "connected": None, "target": None, "source": None, "weight": None})
        return out
    if kind == "search" or (kind == "sim" and case["edges"] > 0.0):
        return None  # whole numbers, or a run whose connectome a search decides
    d = _initial(case, seed)
    p = d["params"]
    x, u, calcium, inp, delta = _activity64(case["n"], case["steps"], p, [(case["n"], p["seed"], p["growth_rate"])], edges=d.get("edges"), x=d.get("x"),
                                            u=d.get("u"), calcium=d.get("calcium"))
    if kind == "activity":
        if case["precision"] == 1:
            x = u = None  # a spike moved by one step is another membrane state altogether
        out = {"x": x, "u": u, "calcium": calcium, "fired": None, "input": None if case["precision"] == 1 else inp, "edges": None}
        for k, name in enumerate(("axons", "dendrites_exc", "dendrites_inh")):
            out[name] = {"grown": None, "delta": delta[k], "connected": None, "vacant": None}
        return out
    if case["n"] < 200000:
        return {"x": None, "u": None, "calcium": calcium, "fired": None, "input": None, "edges": None, "axons": None, "dendrites_exc": None, "dendrites_inh": None}
    return {"calcium": calcium, "fired": None}
