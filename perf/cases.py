"""The work a user of this framework has it do, as timed cases over its public entry points.

``listed()`` names the cases, ``draw(rng)`` makes further ones of the same ranges,
``prepare(case, seed)`` builds what a program has in hand before the call, ``run(state)``
is one pass, ``work(case)`` what the pass cannot do without, and ``exact(case, seed)``
the same outputs in 64 bits from plain torch and numpy statements of the equations.

Kinds:
  sim      one evaluation on a resident ``Simulator``: a generation's parameters (already on the
           GPU), initial state, every timestep, the traces into a device tensor
  run      ``sim.run``: a whole simulation from host arrays to a host array (what a caller of the
           reference's simulator process does)
  batch    ``Batch.run_graph`` over trees of several sizes, one captured run, every member's traces
  score    trace features and the dV/dt peak count of traces that lie on the GPU
  ga       one generation's selection and offspring on the GPU
  predict  the surrogate network's prediction for a generation's offspring
  train    one minibatch step of the surrogate network: loss, gradients, weight update
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from neurogpu_b200 import configs, explore, features
from neurogpu_b200.ga_device import DeviceGA, select_nsga2, select_truncation
from neurogpu_b200.sim import Batch, Model, Simulator, run as run_host
from neurogpu_b200.surrogate import SurrogateMLP

DT = 0.025          # ms, every benchmark configuration's timestep
GA_GENES = 12       # free conductances of the HH fit
N_FEATURES = 20


def listed():
    return [
        # the passive configuration as its script runs it: 128 compartments, 32 sets, 100 ms, host to host
        dict(name="passive_run", kind="run", cell="passive", n_comp=128, sets=32, stims=1, steps=4000, precision="fp32"),
        # a hand-tuning session: a few parameter sets of the HH cell under the three protocols
        dict(name="hh_few", kind="sim", cell="hh", n_comp=500, sets=11, stims=3, steps=400, precision="fp32"),
        # a GA generation of the HH fit at its configuration's population
        dict(name="hh_population", kind="sim", cell="hh", n_comp=500, sets=1024, stims=3, steps=400, precision="fp32"),
        # the HH benchmark batch: a population that fills the GPU
        dict(name="hh_large", kind="sim", cell="hh", n_comp=500, sets=4096, stims=3, steps=200, precision="fp32"),
        # a sensitivity scan of the pyramidal cell: a hundred sets
        dict(name="ttpc_scan", kind="sim", cell="ttpc", n_comp=1501, sets=100, stims=3, steps=200, precision="fp32"),
        # the headline batch of the pyramidal cell
        dict(name="ttpc_large", kind="sim", cell="ttpc", n_comp=1501, sets=4096, stims=3, steps=200, precision="fp32"),
        # the accurate check of a fit's survivors: double precision
        dict(name="hh_double", kind="sim", cell="hh", n_comp=500, sets=256, stims=3, steps=100, precision="fp64"),
        # trees of four sizes in one captured run, five protocols
        dict(name="uneven_batch", kind="batch", sets=4096, stims=5, steps=100),
        # the exploration run's 10,000 traces and a generation's features, in the simulator's own layout
        dict(name="score_10000", kind="score", traces=10000, samples=3168, layout="sample_major"),
        # multi-objective survivors of 5,000 parents and 5,000 offspring, 3 protocols x 20 features, next offspring
        dict(name="ga_nsga2", kind="ga", select="nsga2", n=10000, objectives=60),
        # the screened GA ranks 8,192 offspring under three protocols
        dict(name="mlp_predict", kind="predict", rows=24576, width=512),
        # one training minibatch of that network
        dict(name="mlp_train", kind="train", rows=4096, width=512),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sim", "sim", "sim", "sim", "run", "batch", "score", "ga", "predict", "train"])
    if kind in ("sim", "run"):
        cell = rng.choice(["hh", "hh", "ttpc", "passive"])
        n = {"hh": lambda: _log_int(rng, 120, 1500), "ttpc": lambda: 1501, "passive": lambda: _log_int(rng, 20, 700)}[cell]()
        precision = "fp64" if kind == "sim" and rng.random() < 0.2 else "fp32"
        stims = rng.choice([1, 2, 3, 5])
        # a drawn case stays below the headline batch: compartments x instances, weighed by the type's cost
        room = 1501 * 12288 // (6 if precision == "fp64" else 1) // (n * stims)
        sets = _log_int(rng, 4, max(4, min(5000, room, 1000 if kind == "run" else 5000)))
        steps = rng.randrange(60, 201) if kind == "sim" else rng.randrange(200, 1001)
        if kind == "run":
            steps = max(60, min(steps, 200 * room // max(1, 8 * sets)))
        return dict(kind=kind, cell=cell, n_comp=n, sets=sets, stims=stims, steps=steps, precision=precision)
    if kind == "batch":
        return dict(kind="batch", sets=4 * _log_int(rng, 2, 1000), stims=rng.choice([1, 3, 5]), steps=rng.randrange(40, 101))
    if kind == "score":
        return dict(kind="score", traces=_log_int(rng, 1, 10000), samples=_log_int(rng, 300, 3168),
                    layout=rng.choice(["sample_major", "trace_major"]))
    if kind == "ga":
        return dict(kind="ga", select=rng.choice(["nsga2", "nsga2", "truncation"]), n=_log_int(rng, 64, 10000),
                    objectives=rng.choice([2, 3, 20, 60]))
    if kind == "predict":
        return dict(kind="predict", rows=_log_int(rng, 1, 24576), width=rng.choice([128, 256, 512]))
    return dict(kind="train", rows=_log_int(rng, 128, 4096), width=rng.choice([128, 256, 512]))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _cell(cell, n_comp):
    """The configuration of a cell with one parameter set: its tree, nominal parameters and geometry."""
    if cell == "hh":
        return configs.hh_active(n_sets=1, t_stop=1.0, n_comp=n_comp)
    if cell == "ttpc":
        return configs.ttpc_like(n_sets=1, t_stop=1.0)
    return configs.passive_cable(n_sets=1, t_stop=1.0, n_comp=n_comp)


LEVELS = {"hh": (0.2, 0.5, 1.0, 0.1, 0.7), "ttpc": (0.3, 0.6, 0.9, 0.2, 1.2), "passive": (0.5, 0.1, 1.0, 0.25, 0.75)}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 17)


def _population(cell, w, sets, seed):
    """[sets][params][sections] on the GPU: the configuration's free conductances, each set its own multiples."""
    g = _generator(seed)
    params = torch.from_numpy(w.params).cuda().expand(sets, -1, -1).clone()
    region = np.array([w.cell.region_names[r] for r in w.cell.region])
    if cell == "hh":
        free, lo, hi = configs.MAINEN_FREE, 0.5, 2.0
    elif cell == "ttpc":
        free, lo, hi = configs.TTPC_FREE, 0.1, 10.0
    else:
        free, lo, hi = (("g_pas", ("cable",)),), 0.5, 2.0
    u = torch.rand((sets, len(free)), generator=g, device="cuda")
    mult = lo * (hi / lo) ** u / torch.from_numpy(np.asarray(w.free, dtype=np.float32)).cuda()
    for j, (name, regions) in enumerate(free):
        cols = torch.from_numpy(np.nonzero(np.isin(region, regions))[0]).cuda()
        p = w.cell.mechset.param_index(name)
        params[:, p, cols] = params[:, p, cols] * mult[:, j:j + 1]
    return params.contiguous()


def _stimulus(cell, stims, steps):
    """Current steps that start after 0.5 ms, at the configurations' levels."""
    return configs.step_amps(LEVELS[cell][:stims], steps, DT, 0.5, steps * DT + 1.0)


def _simulator(cell, n_comp, sets, stims, steps, precision, seed):
    w = _cell(cell, n_comp)
    params = _population(cell, w, sets, seed)
    sim = Simulator(Model(w.cell), sets, stims, precision)
    sim.set_params(params)
    sim.set_stimulus(_stimulus(cell, stims, steps), DT, w.stim_node, w.stim_area)
    # soma, middle and last compartment
    sim.set_recording([0, w.cell.n_nodes // 2, w.cell.n_nodes - 1])
    sim.init(w.v_init)
    return sim, params, w.v_init


def _traces(traces, samples, seed):
    """Spike trains on a noisy baseline, [traces][samples] float32, 0.1 ms apart: from silent to bursting."""
    g = _generator(seed)
    t = torch.arange(samples, device="cuda", dtype=torch.float32) * 0.1
    r = torch.rand((6, traces, 1), generator=g, device="cuda")
    isi, start = 6.0 + 60.0 * r[0] ** 2, 0.1 * samples * 0.1 + 20.0 * r[1]
    on = (t >= start) & (t < 0.085 * samples) & (r[2] > 0.15)
    phase = torch.remainder(t - start + 0.03 * (t - start) * r[3], isi)
    v = -70.0 + 6.0 * r[4] + 4.0 * torch.sin(t * (0.02 + 0.05 * r[5]))
    spike = (95.0 + 10.0 * r[4]) * torch.exp(-((phase - 2.0) / 0.45) ** 2) - 9.0 * torch.exp(-((phase - 4.5) / 1.5) ** 2)
    v = v + torch.where(on, spike, torch.zeros_like(spike))
    return (v + 0.2 * torch.randn((traces, samples), generator=g, device="cuda")).contiguous()


def _windows(samples):
    """(stimulus on, stimulus off) ms of a trace of that many samples."""
    return 0.1 * round(0.1 * samples), 0.1 * round(0.85 * samples)


def _objectives(n, m, seed):
    """Errors of a fit's features: correlated through each individual's overall quality."""
    g = _generator(seed)
    quality = torch.rand((n, 1), generator=g, device="cuda", dtype=torch.float64)
    spread = torch.rand((n, m), generator=g, device="cuda", dtype=torch.float64)
    return quality * 2.0 + spread


def _mlp_rows(rows, seed):
    """Network inputs (12 genes and a one-hot protocol) and feature targets."""
    g = _generator(seed)
    x = torch.rand((rows, GA_GENES + 3), generator=g, device="cuda") * 2.0 - 1.0
    x[:, GA_GENES:] = torch.nn.functional.one_hot(torch.arange(rows, device="cuda") % 3, 3).float()
    a = torch.randn((GA_GENES + 3, N_FEATURES), generator=g, device="cuda")
    scale = torch.linspace(0.5, 40.0, N_FEATURES, device="cuda")
    return x, (torch.tanh(x @ a) + 0.05 * torch.randn((rows, N_FEATURES), generator=g, device="cuda")) * scale - 10.0


def _moments(shapes, seed):
    """Adam's first and second moments of a network in mid-training."""
    g = _generator(seed + 5)
    m = [3e-3 * torch.randn(s, generator=g, device="cuda") for s in shapes]
    v = [1e-5 * (0.5 + torch.rand(s, generator=g, device="cuda")) for s in shapes]
    return m, v


STEP_N = 400  # updates the network of a `train` case has behind it


def _network(case, seed):
    x, y = _mlp_rows(case["rows"], seed)
    net = SurrogateMLP(GA_GENES + 3, N_FEATURES, width=case["width"], seed=int(seed) % 1000)
    xs, ys = _mlp_rows(4096, 1)
    net.fit_stats(xs, ys)
    return net, x, y


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sim":
        sim, params, v_init = _simulator(case["cell"], case["n_comp"], case["sets"], case["stims"], case["steps"],
                                         case["precision"], seed)
        return dict(case=case, sim=sim, params=params, v_init=v_init)
    if kind == "run":
        w = _cell(case["cell"], case["n_comp"])
        params = _population(case["cell"], w, case["sets"], seed).cpu().numpy()
        amps = _stimulus(case["cell"], case["stims"], case["steps"])
        return dict(case=case, w=w, model=Model(w.cell), params=params, amps=amps)
    if kind == "batch":
        members = [_simulator("hh", n, case["sets"] // 4, case["stims"], case["steps"], "fp32", seed + k)
                   for k, n in enumerate(BATCH_SIZES)]
        return dict(case=case, batch=Batch([m[0] for m in members]), members=members, stream=torch.cuda.Stream())
    if kind == "score":
        v = _traces(case["traces"], case["samples"], seed)
        if case["layout"] == "sample_major":  # the simulator's trace buffer: consecutive instances of a sample
            v = v.t().contiguous().t()
        return dict(case=case, v=v)
    if kind == "ga":
        g = _generator(seed + 3)
        pop = torch.rand((case["n"], GA_GENES), generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0
        return dict(case=case, obj=_objectives(case["n"], case["objectives"], seed), pop=pop, seed=int(seed),
                    ga=DeviceGA(GA_GENES, eta_c=20.0, eta_m=20.0, cx_prob=0.7, p_mut=0.3, seed=int(seed)))
    net, x, y = _network(case, seed)
    if kind == "train":
        net.m, net.v = _moments([t.shape for t in net.W + net.b], int(seed))
        net.step_n = STEP_N
    return dict(case=case, net=net, x=x, y=y)


BATCH_SIZES = (200, 800, 1500, 3000)


def _read_traces(sim):
    out = torch.empty((sim.n_sets, sim.n_stim, sim.n_rec, sim.n_samples), dtype=torch.float32, device="cuda")
    sim.trace_into(out.data_ptr(), torch.cuda.current_stream())
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sim":
        sim = state["sim"]
        sim.set_params(state["params"])
        sim.init(state["v_init"])
        sim.advance(0, case["steps"])
        return {"v": _read_traces(sim)}
    if kind == "run":
        w = state["w"]
        return {"v": run_host(state["model"], state["params"], state["amps"], DT, w.stim_node, w.stim_area,
                              [0, w.cell.n_nodes // 2, w.cell.n_nodes - 1], w.v_init, case["precision"])}
    if kind == "batch":
        stream = state["stream"]
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for sim, params, _ in state["members"]:
                sim.set_params(params)
            state["batch"].run_graph(state["members"][0][2], case["steps"], case["steps"], stream)
            out = [_read_traces(sim) for sim, _, _ in state["members"]]
        torch.cuda.current_stream().wait_stream(stream)
        return {"v": out}
    if kind == "score":
        on, off = _windows(case["samples"])
        f = features.extract_device(state["v"], 0.1, on, off)
        return {"features": f, "peaks": explore.dvdt_peak_counts(state["v"], stream=torch.cuda.current_stream())}
    if kind == "ga":
        mu = case["n"] // 2
        if case["select"] == "nsga2":
            idx, rank, crowd, fronts = select_nsga2(state["obj"], mu)
            kids = state["ga"].offspring(state["pop"][idx], rank[idx], crowd[idx], mu, 7)
            return {"idx": idx, "rank": rank, "crowd": crowd, "fronts": fronts, "kids": kids}
        score = state["obj"].mean(1)
        idx = select_truncation(score, mu)
        rank = torch.zeros(mu, dtype=torch.int32, device="cuda")
        return {"idx": idx, "kids": state["ga"].offspring(state["pop"][idx], rank, -score[idx], mu, 7)}
    net = state["net"]
    if kind == "predict":
        return {"y": net.predict(state["x"])}
    loss, g_w, g_b = net.loss_and_grads(state["x"], state["y"])
    net.adam_step(g_w, g_b)
    return {"loss": loss, "g_w": list(g_w), "g_b": list(g_b), "w": list(net.W), "b": list(net.b)}


# ------------------------------------------------------------------ work
STATES = {"Ca_HVA": 2, "Ca_LVAst": 2, "CaDynamics_E2": 2, "Ih": 1, "Im": 1, "K_Pst": 2, "K_Tst": 2, "Nap_Et2": 2,
          "NaTa_t": 2, "NaTs2_t": 2, "SK_E2": 1, "SKv3_1": 1, "ca": 2, "cad": 2, "kca": 1, "km": 1, "kv": 1, "na": 2}
ON_CHIP = 126e6  # bytes of L2: a batch whose state fits need not leave it between steps


def _sim_work(cell, n_comp, sets, stims, steps, width):
    """Parameters in, traces out; a state (V and channel states, read and written) that exceeds the
    L2 moves every step.  Operations: 24 a compartment for the solve, 24 a channel state."""
    c = _cell(cell, n_comp).cell
    states = sum(STATES.get(m, 0) * int(c.mech_mask[k].sum()) for k, m in enumerate(c.mechset.mechs))
    inst = sets * stims
    state_bytes = float(inst) * (c.n_nodes + states) * width
    io = 4.0 * (sets * c.mechset.n_params * c.n_sections + inst * 3 * steps + stims * steps)
    return dict(bytes=io + (2.0 * state_bytes * steps if state_bytes > ON_CHIP else 0.0),
                flops=24.0 * inst * steps * (c.n_nodes + states))


def work(case):
    kind = case["kind"]
    if kind in ("sim", "run"):
        return _sim_work(case["cell"], case["n_comp"], case["sets"], case["stims"], case["steps"],
                         8 if case["precision"] == "fp64" else 4)
    if kind == "batch":
        each = [_sim_work("hh", n, case["sets"] // 4, case["stims"], case["steps"], 4) for n in BATCH_SIZES]
        return dict(bytes=sum(e["bytes"] for e in each), flops=sum(e["flops"] for e in each))
    if kind == "score":
        n = case["traces"] * case["samples"]
        return dict(bytes=4.0 * n + 84.0 * case["traces"], flops=12.0 * n)
    if kind == "ga":
        n, m, mu = case["n"], case["objectives"], case["n"] // 2
        return dict(bytes=8.0 * n * m + 8.0 * GA_GENES * 2 * mu + 24.0 * n, flops=float(n) * m * math.log2(max(n, 2)))
    rows, width, n_in = case["rows"], case["width"], GA_GENES + 3
    weights = n_in * width + 2 * width * width + width * N_FEATURES
    if kind == "predict":
        return dict(bytes=4.0 * rows * (n_in + N_FEATURES) + 2.0 * weights, flops=2.0 * rows * weights)
    return dict(bytes=4.0 * rows * (n_in + N_FEATURES) + 28.0 * weights, flops=6.0 * rows * weights)


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind in ("sim", "run"):
        w = _cell(case["cell"], case["n_comp"])
        params = _population(case["cell"], w, case["sets"], seed)
        return {"v": _exact_simulation(w, params, _stimulus(case["cell"], case["stims"], case["steps"]))}
    if kind == "batch":
        out = []
        for k, n in enumerate(BATCH_SIZES):
            w = _cell("hh", n)
            out.append(_exact_simulation(w, _population("hh", w, case["sets"] // 4, seed + k),
                                         _stimulus("hh", case["stims"], case["steps"])))
        return {"v": out}
    if kind == "score":
        v = _traces(case["traces"], case["samples"], seed)
        return {"features": _exact_features(v, *_windows(case["samples"])), "peaks": None}
    if kind == "ga":
        return _exact_ga(case, seed)
    return _exact_network(case, seed)


def _exact_simulation(w, params, amps):
    """The step in double: implicit Euler of the branched cable with currents at the old voltage
    (recorded first), then channel states over dt at the new voltage.  Nodes are ordered by depth,
    so that a depth is a slice of every array; arrays are [node][set][protocol]."""
    c = w.cell
    n, dev, f8 = c.n_nodes, torch.device("cuda"), torch.float64
    depth = np.zeros(n, dtype=np.int64)
    for i in range(1, n):
        depth[i] = depth[c.parent[i]] + 1
    order = np.argsort(depth, kind="stable")
    place = np.empty(n, dtype=np.int64)
    place[order] = np.arange(n)
    cuts = np.searchsorted(depth[order], np.arange(depth.max() + 2))
    up = np.where(c.parent[order] >= 0, place[np.maximum(c.parent[order], 0)], 0)
    sets, stims, steps = params.shape[0], amps.shape[0], amps.shape[1]

    def column(x):
        return torch.from_numpy(np.asarray(x, dtype=np.float64)[order]).to(dev)[:, None, None]

    a, b, cm = column(c.a), column(c.b), column(c.cm)
    up_t = torch.from_numpy(up).to(dev)
    section = torch.from_numpy(np.asarray(c.section, dtype=np.int64)[order]).to(dev)
    dt = float(np.float32(DT))
    axial = -a.expand(n, 1, 1).clone()
    axial[0] = 0.0
    axial.index_add_(0, up_t[1:], -b[1:])
    p8 = params.double()
    mech_nodes, p_of = {}, {}
    for k, name in enumerate(c.mechset.mechs):
        where = torch.from_numpy(np.nonzero(np.asarray(c.mech_mask[k])[order])[0]).to(dev)
        if where.numel():
            mech_nodes[name] = where
            for p in c.mechset.mech_params[k]:
                p_of[c.mechset.params[p]] = p8[:, p, :][:, section[where]].t()[:, :, None].contiguous()
    channels = _MAINEN if c.mechset.name == "mainen" else _TTPC
    shape = (n, sets, stims)
    v = torch.full(shape, float(np.float32(w.v_init)), dtype=f8, device=dev)
    st = {}
    cur, cond = channels(mech_nodes, p_of, v, st, None)
    amp = torch.from_numpy(amps.astype(np.float64)).to(dev) * (100.0 / float(np.float32(w.stim_area)))
    sites = torch.from_numpy(place[np.array([0, n // 2, n - 1])]).to(dev)
    stim = int(place[w.stim_node])
    out = torch.empty((sets, stims, 3, steps), dtype=torch.float64, device=dev)
    slices = [(int(cuts[d]), int(cuts[d + 1])) for d in range(len(cuts) - 1)]
    for t in range(steps):
        out[..., t] = v[sites].permute(1, 2, 0)
        diag = cond + (cm / (1000.0 * dt)) + axial
        dv = v[up_t] - v
        dv[0] = 0.0
        rhs = -cur - a * dv
        rhs.index_add_(0, up_t[1:], (b * dv)[1:])
        rhs[stim] += amp[None, :, t]
        for lo, hi in reversed(slices[1:]):
            f = b[lo:hi] / diag[lo:hi]
            diag.index_add_(0, up_t[lo:hi], -f * a[lo:hi])
            rhs.index_add_(0, up_t[lo:hi], -f * rhs[lo:hi])
        x = rhs
        x[0] /= diag[0]
        for lo, hi in slices[1:]:
            x[lo:hi] = (rhs[lo:hi] - a[lo:hi] * x[up_t[lo:hi]]) / diag[lo:hi]
        v = v + x
        cur, cond = channels(mech_nodes, p_of, v, st, dt)
    return out


def _vtrap(z):
    """z / (e^z - 1)"""
    return torch.where(z == 0, torch.ones_like(z), z / torch.expm1(z))


class _Channels:
    """Sums of the currents and conductances of a set's channels; gates take an exponential step."""

    def __init__(self, nodes, v, st, dt):
        self.nodes, self.v, self.st, self.dt = nodes, v, st, dt
        self.cur, self.cond = torch.zeros_like(v), torch.zeros_like(v)

    def gate(self, name, inf, rate):
        if self.dt is None:
            self.st[name] = inf
        else:
            x = self.st[name]
            self.st[name] = x - torch.expm1(-self.dt * rate) * (inf - x)
        return self.st[name]

    def ab(self, name, alpha, beta, q):
        return self.gate(name, alpha / (alpha + beta), q * (alpha + beta))

    def add(self, mech, g, e):
        i = g * (self.v[self.nodes[mech]] - e)
        self.cur.index_add_(0, self.nodes[mech], i)
        self.cond.index_add_(0, self.nodes[mech], g.expand_as(i).contiguous())
        return i


def _calcium_potential(cai, celsius):
    return 1000.0 * 8.3134 * (celsius + 273.15) / 96485.309 / 2.0 * torch.log(2.0 / cai)


def _spread(values, at, to, like):
    """`values` on nodes `at`, taken at nodes `to` (a subset)."""
    full = torch.zeros_like(like)
    full[at] = values
    return full[to]


def _MAINEN(nodes, p, v, st, dt):
    """The cortical set of Mainen and Sejnowski: ca, cad, kca, km, kv, na and the leak (37 C)."""
    q, ch = 2.3 ** 1.4, _Channels(nodes, v, st, dt)
    if "ca" in nodes:
        u = v[nodes["ca"]]
        m = ch.ab("ca_m", 0.209 * _vtrap(-(u + 27.0) / 3.8), 0.94 * torch.exp((-75.0 - u) / 17.0), q)
        h = ch.ab("ca_h", 0.000457 * torch.exp((-13.0 - u) / 50.0), 0.0065 / (torch.exp((-u - 15.0) / 28.0) + 1.0), q)
    if "cad" in nodes:
        if dt is None:
            st["cai"] = torch.full_like(v[nodes["cad"]], 1e-4)
        else:
            drive = (-10000.0 / (2.0 * 96485.309 * 0.09334562733124982) * st["ica"]).clamp(min=0.0)
            ch.gate("cai", (drive + 1e-4 / 200.0) * 200.0, torch.full_like(drive, 1.0 / 200.0))
    if "kca" in nodes:
        cai = _spread(st["cai"], nodes["cad"], nodes["kca"], v)
        kn = ch.ab("kca_n", p["Ra_kca"] * cai ** p["caix_kca"], p["Rb_kca"], q)
        ch.add("kca", 1e-4 * q * p["gbar_kca"] * kn, -90.0)
    for k in ("km", "kv"):
        if k in nodes:
            z = (v[nodes[k]] - p[f"tha_{k}"]) / p[f"qa_{k}"]
            kn = ch.ab(k, p[f"Ra_{k}"] * p[f"qa_{k}"] * _vtrap(-z), p[f"Rb_{k}"] * p[f"qa_{k}"] * _vtrap(z), q)
            ch.add(k, 1e-4 * q * p[f"gbar_{k}"] * kn, -90.0)
    if "na" in nodes:
        u = v[nodes["na"]] - 5.0
        z = (u - p["tha_na"]) / p["qa_na"]
        m3 = ch.ab("na_m", p["Ra_na"] * p["qa_na"] * _vtrap(-z), p["Rb_na"] * p["qa_na"] * _vtrap(z), q) ** 3
        rate = p["Rd_na"] * p["qi_na"] * _vtrap(-(u - p["thi1_na"]) / p["qi_na"]) \
            + p["Rg_na"] * p["qi_na"] * _vtrap((u - p["thi2_na"]) / p["qi_na"])
        hn = ch.gate("na_h", 1.0 / (1.0 + torch.exp((u - p["thinf_na"]) / p["qinf_na"])), q * rate)
        ch.add("na", 1e-4 * q * p["gbar_na"] * m3 * hn, 60.0)
    if "ca" in nodes:
        cai = _spread(st["cai"], nodes["cad"], nodes["ca"], v)
        st["ica"] = ch.add("ca", 1e-4 * q * p["gbar_ca"] * m * m * h, _calcium_potential(cai, 37.0))
        st["ica"] = _spread(st["ica"], nodes["ca"], nodes["cad"], v)
    ch.add("pas", p["g_pas"].expand_as(v[nodes["pas"]]), p["e_pas"])
    return ch.cur, ch.cond


def _TTPC(nodes, p, v, st, dt):
    """The thick-tufted pyramidal cell's set (34 C)."""
    q, ch = 2.3 ** 1.3, _Channels(nodes, v, st, dt)
    gates = {}

    def sig(z):
        return 1.0 / (1.0 + torch.exp(z))

    if "Ca_HVA" in nodes:
        u = v[nodes["Ca_HVA"]]
        m = ch.ab("hva_m", 0.055 * 3.8 * _vtrap((-27.0 - u) / 3.8), 0.94 * torch.exp((-75.0 - u) / 17.0), 1.0)
        h = ch.ab("hva_h", 0.000457 * torch.exp((-13.0 - u) / 50.0), 0.0065 * sig((-u - 15.0) / 28.0), 1.0)
        gates["Ca_HVA"] = p["gCa_HVAbar_Ca_HVA"] * m * m * h
    if "Ca_LVAst" in nodes:
        u = v[nodes["Ca_LVAst"]] + 10.0
        m = ch.gate("lva_m", sig((u + 30.0) / -6.0), q / (5.0 + 20.0 * sig((u + 25.0) / 5.0)))
        h = ch.gate("lva_h", sig((u + 80.0) / 6.4), q / (20.0 + 50.0 * sig((u + 40.0) / 7.0)))
        gates["Ca_LVAst"] = p["gCa_LVAstbar_Ca_LVAst"] * m * m * h
    if "CaDynamics_E2" in nodes:
        at = nodes["CaDynamics_E2"]
        if dt is None:
            st["cai"] = torch.full_like(v[at], 5e-5)
        else:
            decay = p["decay_CaDynamics_E2"]
            inf = (-10000.0 / (2.0 * 96485.309) * st["ica"] * p["gamma_CaDynamics_E2"] / p["depth_CaDynamics_E2"]
                   + p["minCai_CaDynamics_E2"] / decay) * decay
            ch.gate("cai", inf, 1.0 / decay)
    if "Ih" in nodes:
        u = v[nodes["Ih"]]
        m = ch.ab("ih", 0.001 * 6.43 * 11.9 * _vtrap((u + 154.9) / 11.9), 0.193 * torch.exp(u / 33.1), 1.0)
        ch.add("Ih", p["gIhbar_Ih"] * m, p["ehcn_Ih"])
    if "Im" in nodes:
        u = v[nodes["Im"]] + 35.0
        m = ch.ab("im", 3.3e-3 * torch.exp(0.1 * u), 3.3e-3 * torch.exp(-0.1 * u), q)
        ch.add("Im", p["gImbar_Im"] * m, -85.0)
    if "K_Pst" in nodes:
        u = v[nodes["K_Pst"]] + 10.0
        tau = torch.where(u < -50.0, 1.25 + 175.03 * torch.exp(0.026 * u), 1.25 + 13.0 * torch.exp(-0.026 * u))
        m = ch.gate("kp_m", sig(-(u + 1.0) / 12.0), q / tau)
        h = ch.gate("kp_h", sig((u + 54.0) / 11.0),
                    q / (360.0 + (1010.0 + 24.0 * (u + 55.0)) * torch.exp(-((u + 75.0) / 48.0) ** 2)))
        ch.add("K_Pst", p["gK_Pstbar_K_Pst"] * m * m * h, -85.0)
    if "K_Tst" in nodes:
        u = v[nodes["K_Tst"]] + 10.0
        m = ch.gate("kt_m", sig(-u / 19.0), q / (0.34 + 0.92 * torch.exp(-((u + 71.0) / 59.0) ** 2)))
        h = ch.gate("kt_h", sig((u + 66.0) / 10.0), q / (8.0 + 49.0 * torch.exp(-((u + 73.0) / 23.0) ** 2)))
        ch.add("K_Tst", p["gK_Tstbar_K_Tst"] * m ** 4 * h, -85.0)
    if "Nap_Et2" in nodes:
        u = v[nodes["Nap_Et2"]]
        z = (u + 38.0) / 6.0
        m = ch.gate("nap_m", sig((u + 52.6) / -4.6), q / 6.0 * (0.182 * 6.0 * _vtrap(-z) + 0.124 * 6.0 * _vtrap(z)))
        h = ch.gate("nap_h", sig((u + 48.8) / 10.0), q * (2.88e-6 * 4.63 * _vtrap((u + 17.0) / 4.63)
                                                          + 6.94e-6 * 2.63 * _vtrap(-(u + 64.4) / 2.63)))
        ch.add("Nap_Et2", p["gNap_Et2bar_Nap_Et2"] * m ** 3 * h, 50.0)
    for mech, key, th_m, th_h in (("NaTa_t", "gNaTa_tbar_NaTa_t", -38.0, -66.0),
                                  ("NaTs2_t", "gNaTs2_tbar_NaTs2_t", -32.0, -60.0)):
        if mech in nodes:
            u = v[nodes[mech]]
            z, y = (u - th_m) / 6.0, (u - th_h) / 6.0
            m = ch.ab(mech + "_m", 0.182 * 6.0 * _vtrap(-z), 0.124 * 6.0 * _vtrap(z), q)
            h = ch.ab(mech + "_h", 0.015 * 6.0 * _vtrap(y), 0.015 * 6.0 * _vtrap(-y), q)
            ch.add(mech, p[key] * m ** 3 * h, 50.0)
    ch.add("pas", p["g_pas"].expand_as(v[nodes["pas"]]), p["e_pas"])
    if "SK_E2" in nodes:
        cai = _spread(st["cai"], nodes["CaDynamics_E2"], nodes["SK_E2"], v)
        cai = torch.where(cai < 1e-7, cai + 1e-7, cai)
        z = ch.gate("sk", 1.0 / (1.0 + (0.00043 / cai) ** 4.8), 1.0 / p["zTau_SK_E2"])
        ch.add("SK_E2", p["gSK_E2bar_SK_E2"] * z, -85.0)
    if "SKv3_1" in nodes:
        u = v[nodes["SKv3_1"]]
        m = ch.gate("skv", sig((u - 18.7) / -9.7), (1.0 + torch.exp((u + 46.56) / -44.14)) / 4.0)
        ch.add("SKv3_1", p["gSKv3_1bar_SKv3_1"] * m, -85.0)
    if gates:
        at = nodes["CaDynamics_E2"]
        ica = torch.zeros_like(v)
        for mech, g in gates.items():
            e = _calcium_potential(_spread(st["cai"], at, nodes[mech], v), 34.0)
            ica.index_add_(0, nodes[mech], ch.add(mech, g, e))
        st["ica"] = ica[at]
    return ch.cur, ch.cond


def _exact_features(v, on, off, threshold=-20.0, dt=0.1):
    """The 20 features of every trace in double, from their definitions."""
    n, t = v.shape
    v = v.double()
    i0, i1 = int(round(on / dt)), min(t, int(round(off / dt)))
    w, dur = v[:, i0:i1], (i1 - i0) * dt
    up = torch.zeros_like(w, dtype=torch.bool)
    up[:, 1:] = (w[:, :-1] < threshold) & (w[:, 1:] >= threshold)
    count = up.sum(1)
    has1, has2 = count >= 1, count >= 2
    seg = torch.cumsum(up, 1)
    k = max(2, int(count.max())) + 1
    at = torch.arange(w.shape[1], device=v.device, dtype=torch.float64).expand_as(w) * dt
    when = torch.full((n, k), math.inf, dtype=torch.float64, device=v.device)
    when = when.scatter_reduce(1, torch.where(up, seg - 1, torch.full_like(seg, k - 1)),
                               torch.where(up, at, torch.full_like(at, math.inf)), "amin")[:, :k - 1]
    isi = when[:, 1:] - when[:, :-1]
    ok = torch.isfinite(isi)
    isi0 = torch.where(ok, isi, torch.zeros_like(isi))
    ni = (count - 1).clamp(min=1).double()
    full = torch.full((n,), dur, dtype=torch.float64, device=v.device)
    mean_isi = torch.where(has2, isi0.sum(1) / ni, full)
    dev = torch.where(ok, isi - mean_isi[:, None], torch.zeros_like(isi))
    cv = torch.where(has2, (dev.square().sum(1) / ni).sqrt() / mean_isi, torch.zeros_like(full))
    last_isi = isi0.gather(1, (count - 2).clamp(min=0)[:, None])[:, 0]
    first = torch.where(has1, when[:, 0], full)
    last = torch.where(has1, when.gather(1, (count - 1).clamp(min=0)[:, None])[:, 0], full)
    peak = torch.full((n, k + 1), -math.inf, dtype=torch.float64, device=v.device).scatter_reduce(1, seg, w, "amax")[:, 1:]
    low = torch.full((n, k + 1), math.inf, dtype=torch.float64, device=v.device).scatter_reduce(1, seg, w, "amin")[:, 1:]
    has = torch.isfinite(peak)
    c1 = count.clamp(min=1).double()
    zero = torch.zeros_like(peak)
    pk = torch.where(has1, torch.where(has, peak, zero).sum(1) / c1, w.max(1).values)
    sd = torch.where(has1, (torch.where(has, peak - pk[:, None], zero).square().sum(1) / c1).sqrt(), torch.zeros_like(pk))
    ahp = torch.where(has1, torch.where(has, low, zero).sum(1) / c1, w.min(1).values)
    above = ((w >= (0.5 * (pk + ahp))[:, None]) & (seg > 0)).sum(1) * dt
    nul, one = torch.zeros_like(pk), torch.ones_like(pk)

    def mean(a, b):
        ia = max(0, int(round(a / dt)))
        return v[:, ia:min(t, max(ia + 1, int(round(b / dt))))].mean(1)

    after = mean(off + 10.0, t * dt) if off + 10.0 < t * dt else v[:, -1]
    return torch.stack([count.double(), first, mean_isi, cv, torch.where(has2, isi0[:, 0], full),
                        torch.where(has2, last_isi, full), torch.where(has2, last_isi / isi0[:, 0].clamp(min=1e-6), one),
                        pk, sd, ahp, pk - ahp, torch.where(has1, above / c1, nul), mean(max(0.0, on - 10.0), on),
                        mean(max(on, off - 50.0), off), after, v.max(1).values, w.min(1).values, w.mean(1), w.std(1),
                        last], 1)


def _splitmix(x):
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _exact_ga(case, seed):
    """Survivors by non-dominated sorting and crowding (Deb et al. 2002) or by score, then
    tournament, bounded SBX and polynomial mutation on a SplitMix64 stream."""
    n, m, mu = case["n"], case["objectives"], case["n"] // 2
    obj = _objectives(n, m, seed)
    g = _generator(seed + 3)
    pop = (torch.rand((n, GA_GENES), generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0).cpu().numpy()
    if case["select"] == "truncation":
        score = obj.mean(1).cpu().numpy()
        idx = np.argsort(score, kind="stable")[:mu]
        return {"idx": None, "kids": _exact_offspring(pop[idx], np.zeros(mu, np.int32), -score[idx], mu, seed)}
    dominated = torch.empty((n, n), dtype=torch.bool, device="cuda")  # [j][i]: j dominates i
    for j in range(0, n, 250):
        le = torch.ones((min(250, n - j), n), dtype=torch.bool, device="cuda")
        lt = torch.zeros_like(le)
        for k in range(m):
            le &= obj[j:j + 250, k, None] <= obj[None, :, k]
            lt |= obj[j:j + 250, k, None] < obj[None, :, k]
        dominated[j:j + 250] = le & lt
    rank = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    left = torch.ones(n, dtype=torch.bool, device="cuda")
    by = dominated.sum(0, dtype=torch.int32)
    front = 0
    while bool(left.any()):
        now = left & (by == 0)
        rank[now] = front
        left &= ~now
        by -= dominated[now].sum(0, dtype=torch.int32)
        front += 1
    rank, f = rank.cpu().numpy(), obj.cpu().numpy()
    crowd = np.zeros(n)
    for r in range(front):
        who = np.nonzero(rank == r)[0]
        for k in range(m):
            at = who[np.argsort(f[who, k], kind="stable")]
            fk = f[at, k]
            crowd[at[0]] = crowd[at[-1]] = np.inf
            if len(at) > 2 and fk[-1] > fk[0]:
                crowd[at[1:-1]] += (fk[2:] - fk[:-2]) / (fk[-1] - fk[0])
    idx = np.lexsort((np.arange(n), -crowd, rank))[:mu]
    return {"idx": None, "rank": None, "crowd": crowd, "fronts": None,
            "kids": _exact_offspring(pop[idx], rank[idx], crowd[idx], mu, seed)}


def _exact_offspring(pop, rank, crowd, kids, seed, generation=7, eta=20.0, cx=0.7, p_mut=0.3, lo=-1.0, hi=1.0):
    key = _splitmix(np.uint64(int(seed)) ^ _splitmix(np.uint64(generation)))
    child = np.arange(kids, dtype=np.uint64) << np.uint64(20)

    def bits(d):
        return _splitmix(key ^ _splitmix(child | np.uint64(d)))

    def uniform(d):
        return (bits(d) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53

    def pick(d):
        return (((bits(d) >> np.uint64(32)) * np.uint64(len(pop))) >> np.uint64(32)).astype(np.int64)

    def best(i, j):
        return np.where((rank[j] < rank[i]) | ((rank[j] == rank[i]) & (crowd[j] > crowd[i])), j, i)

    x, y = pop[best(pick(0), pick(1))], pop[best(pick(2), pick(3))]
    mate, first = uniform(4) < cx, uniform(5) < 0.5
    out = np.empty((kids, pop.shape[1]))
    with np.errstate(all="ignore"):
        for k in range(pop.shape[1]):
            d = 6 + 5 * k
            a, b, u = x[:, k], y[:, k], uniform(d + 1)
            x1, x2 = np.minimum(a, b), np.maximum(a, b)

            def spread(beta):
                alpha = 2.0 - beta ** -(eta + 1.0)
                return np.where(u <= 1.0 / alpha, (u * alpha) ** (1.0 / (eta + 1.0)),
                                (1.0 / (2.0 - u * alpha)) ** (1.0 / (eta + 1.0)))

            y1 = np.clip(0.5 * (x1 + x2 - spread(1.0 + 2.0 * (x1 - lo) / (x2 - x1)) * (x2 - x1)), lo, hi)
            y2 = np.clip(0.5 * (x1 + x2 + spread(1.0 + 2.0 * (hi - x2) / (x2 - x1)) * (x2 - x1)), lo, hi)
            crossed = (uniform(d) < 0.5) & (np.abs(a - b) > 1e-14)
            val = np.where(crossed, np.where(first != (uniform(d + 2) < 0.5), y1, y2), np.where(first, a, b))
            val = np.where(mate, val, a)
            r = uniform(d + 4)
            d1, d2 = (val - lo) / (hi - lo), (hi - val) / (hi - lo)
            dq = np.where(r < 0.5, (2.0 * r + (1.0 - 2.0 * r) * (1.0 - d1) ** (eta + 1.0)) ** (1.0 / (eta + 1.0)) - 1.0,
                          1.0 - (2.0 * (1.0 - r) + 2.0 * (r - 0.5) * (1.0 - d2) ** (eta + 1.0)) ** (1.0 / (eta + 1.0)))
            out[:, k] = np.where(uniform(d + 3) < p_mut, np.clip(val + dq * (hi - lo), lo, hi), val)
    return out


def _exact_network(case, seed):
    """The network (three GELU layers in tanh form) in double: its prediction, or the loss, the
    gradients and the weights after one Adam step."""
    width, n_in, n_out = case["width"], GA_GENES + 3, N_FEATURES
    x, y = (t.double() for t in _mlp_rows(case["rows"], seed))
    xs, ys = (t.double() for t in _mlp_rows(4096, 1))
    xn = (x - xs.mean(0)) / xs.std(0).clamp(min=1e-6)
    y_mu, y_sd = ys.mean(0), ys.std(0).clamp(min=1e-6)
    g = torch.Generator(device="cpu").manual_seed(int(seed) % 1000)
    k_in, k_out = 64, 32  # the padded widths
    w = []
    for k, (rows, cols) in enumerate([(width, k_in), (width, width), (width, width), (k_out, width)]):
        t = torch.randn(rows, cols, generator=g) / math.sqrt(n_in if k == 0 else width)
        if k == 0:
            t[:, n_in:] = 0.0
        if k == 3:
            t[n_out:, :] = 0.0
        w.append(t.cuda().double().requires_grad_(True))
    b = [torch.zeros(t.shape[0], dtype=torch.float64, device="cuda", requires_grad=True) for t in w]
    h = torch.nn.functional.pad(xn, (0, k_in - n_in))
    for k in range(3):
        h = torch.nn.functional.gelu(h @ w[k].t() + b[k], approximate="tanh")
    out = (h @ w[3].t() + b[3])[:, :n_out]
    if case["kind"] == "predict":
        return {"y": (out * y_sd + y_mu).detach()}
    loss = (out - (y - y_mu) / y_sd).square().sum() / (case["rows"] * n_out)
    grads = torch.autograd.grad(loss, w + b)
    m, v = _moments([t.shape for t in w + b], int(seed))
    n, new = STEP_N + 1, []
    for t, gr, mm, vv in zip(w + b, grads, m, v):
        mm, vv = 0.9 * mm.double() + 0.1 * gr, 0.999 * vv.double() + 0.001 * gr * gr
        new.append((t - 1e-3 * (mm / (1 - 0.9 ** n)) / ((vv / (1 - 0.999 ** n)).sqrt() + 1e-8)).detach())
    new[0][:, n_in:] = 0.0
    new[3][n_out:, :] = 0.0
    new[7][n_out:] = 0.0
    return {"loss": loss.detach(), "g_w": list(grads[:4]), "g_b": list(grads[4:]), "w": new[:4], "b": new[4:]}
