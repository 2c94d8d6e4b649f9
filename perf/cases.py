"""The work users bring to this framework, as timed cases.

A case is a dict of plain values.  `listed()` names the fixed ones, `draw`
gives others of the same ranges, `prepare` builds what a program holds before
the call (a prepared network, a fitting problem, a network with its training
set), `run` is one pass through the public entry points with everything the
user reads back, `work` the bytes and operations the pass cannot do without
and `exact` the same results in 64 bits without this package.

Kinds:

- ``net``    a CUBA network (examples/misc/CUBA.py of the reference) through
             Connections (zero delay), DelayConnections or Synapses, run for
             `steps` steps with a SpikeMonitor; the spikes and the state are
             read after the run
- ``coba``   the same with conductance synapses: a nonlinear model, so the
             update is generated code (Euler, RK2 or exponential Euler)
- ``batch``  many small CUBA networks side by side in a NetworkBatch
- ``stdp``   Poisson inputs onto LIF outputs, all to all, ExponentialSTDP
             (examples/plasticity/STDP1.py of the reference, scaled up);
             weights, traces, spikes and states are read after the run
- ``fit``    one evaluation of every candidate of a fitting problem (the
             inner call of every optimiser)
- ``fitcall`` a whole modelfitting() call
- ``grad``   forward and backward of the proposal network on one batch
- ``train``  epochs of training of the proposal network
"""
import math

import numpy as np
import torch

import brian_b200 as b
from brian_b200 import Hz, mV, ms
from brian_b200._lib import MLP_COLS, MLP_ROWS, MLPHandle
from brian_b200.modelfitting import PSO, FittingProblem, modelfitting
from brian_b200.synthetic import PARAMS, PRIOR, RESET, THRESHOLD, FitWorkload, adaptive_lif_equations

DT = 1e-4
TAUM, TAUE, TAUI = 20 * ms, 5 * ms, 10 * ms
EL, VT, VR = -49 * mV, -50 * mV, -60 * mV
EE, EI = 0 * mV, -80 * mV          # reversal potentials of the conductance form
YDIM = 5


def listed():
    return [
        # the shortest call: a small network advanced by 10 ms (a user stepping through a protocol)
        dict(name="cuba-1000", kind="net", via="connection", n=1000, indegree=80, steps=100, precision=64),
        # the plain benchmark network of the reference, half a second
        dict(name="cuba-4000", kind="net", via="connection", n=4000, indegree=80, steps=5000, precision=64),
        # conductance synapses: generated code (the reference's COBA example), Euler
        dict(name="coba-4000", kind="coba", n=4000, indegree=80, steps=1000, method="Euler"),
        # heterogeneous delays at an ordinary, odd size, FP32 state
        dict(name="cuba-delay-10007", kind="net", via="delay", n=10007, indegree=200, steps=2000, precision=32),
        # the headline network of the benchmark
        dict(name="cuba-delay-262144", kind="net", via="delay", n=262144, indegree=1000, steps=5000, precision=64),
        # per-synapse weights and delays through Synapses, the benchmark's smaller size
        dict(name="cuba-synapses-32768", kind="net", via="synapses", n=32768, indegree=160, steps=1000, precision=64),
        # a parameter study: one network per SM, the benchmark's batch
        dict(name="batch-148x4000", kind="batch", count=148, n=4000, indegree=80, steps=5000),
        # the benchmark's plasticity network
        dict(name="stdp-10000x4096", kind="stdp", nin=10000, nout=4096, steps=5000),
        # the benchmark's fitting shape: inputs of 1-20 s, 1024 candidates per target
        dict(name="fit-64x1024", kind="fit", targets=64, particles=1024, seconds=20.0, precision="float",
             method="Euler"),
        # a whole fit as the reference's users call it: double precision, a short recording, few targets
        dict(name="fitcall-2x1000", kind="fitcall", targets=2, particles=1000, seconds=2.0, precision="double",
             method="Euler", iterations=5),
        # one data-parallel training step's gradients at the default batch of the proposal network
        dict(name="grad-4096", kind="grad", batch=4096),
        # training at the benchmark's batch
        dict(name="train-16384", kind="train", rows=131072, batch=16384, epochs=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["net", "net", "net", "net", "coba", "batch", "stdp", "fit", "fitcall", "grad", "train"])
    if kind == "net":
        via = rng.choice(["connection", "delay", "synapses"])
        n = _log_int(rng, 600, {"connection": 8000, "delay": 200000, "synapses": 60000}[via])
        # the work of a drawn network stays below the largest listed one of its kind
        indegree = min(n // 8, _log_int(rng, 40, 600 if via == "delay" else 160))
        return dict(kind="net", via=via, n=n, indegree=indegree, steps=_log_int(rng, 100, 2000),
                    precision=rng.choice([64, 64, 32]) if via != "synapses" else 64)
    if kind == "coba":
        return dict(kind="coba", n=_log_int(rng, 800, 8000), indegree=_log_int(rng, 40, 100),
                    steps=_log_int(rng, 100, 1000), method=rng.choice(["Euler", "RK", "exponential_Euler"]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 148), n=_log_int(rng, 500, 4000), indegree=_log_int(rng, 40, 80),
                    steps=_log_int(rng, 100, 1000))
    if kind == "stdp":
        return dict(kind="stdp", nin=_log_int(rng, 500, 10000), nout=_log_int(rng, 64, 4096),
                    steps=_log_int(rng, 500, 4000))
    if kind == "fit":
        return dict(kind="fit", targets=_log_int(rng, 1, 64), particles=_log_int(rng, 100, 1024),
                    seconds=round(rng.uniform(2.0, 20.0), 2), precision=rng.choice(["float", "double"]),
                    method=rng.choice(["Euler", "Euler", "RK", "exponential_Euler"]))
    if kind == "fitcall":
        return dict(kind="fitcall", targets=rng.randint(1, 8), particles=_log_int(rng, 100, 1000),
                    seconds=round(rng.uniform(1.0, 2.0), 2), precision=rng.choice(["float", "double"]),
                    method="Euler", iterations=rng.randint(2, 5))
    batch = 512 * _log_int(rng, 1, 32)
    if kind == "grad":
        return dict(kind="grad", batch=batch)
    return dict(kind="train", rows=batch * rng.randint(2, 8) + rng.randint(0, 511), batch=batch,
                epochs=rng.randint(1, 4))


# ---------------------------------------------------------------- networks
def _device():
    return torch.device("cuda:0")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _rows(n_src, n_tgt, k, gen):
    """Connectivity in which every target has k distinct sources, as CSR rows
    per source (targets ascending): one source from each of k equal strata."""
    k = max(1, min(k, n_src))
    u = torch.rand((n_tgt, k), generator=gen, device=_device(), dtype=torch.float64)
    lo = torch.arange(k, device=_device(), dtype=torch.float64)
    src = ((lo + u) * (n_src / k)).floor_().to(torch.int64)
    first = torch.ceil(lo * (n_src / k) - 1e-9).to(torch.int64)      # strata do not share a source
    src = torch.minimum(torch.maximum(src, first), torch.cat([first[1:] - 1, first.new_tensor([n_src - 1])]))
    del u
    key = (src * n_tgt).add_(torch.arange(n_tgt, device=_device()).reshape(-1, 1)).reshape(-1)
    del src
    key = torch.sort(key)[0]
    cols = (key % n_tgt).to(torch.int32)
    rows = key.div_(n_tgt, rounding_mode="floor")
    rowptr = torch.zeros(n_src + 1, dtype=torch.int64, device=_device())
    torch.cumsum(torch.bincount(rows, minlength=n_src), 0, out=rowptr[1:])
    return rowptr, cols


def _wiring(c, seed):
    """Connectivity, weights, delays and initial v of one network, on the GPU."""
    gen = _generator(seed)
    n, k = c["n"], c["indegree"]
    ne = int(0.8 * n)
    ke = max(1, int(0.8 * k))
    via = c.get("via", "connection")
    d = {"n": n, "ne": ne}
    for name, cnt, kk in (("e", ne, ke), ("i", n - ne, max(1, k - ke))):
        d["row" + name], d["col" + name] = _rows(cnt, n, kk, gen)
        m = len(d["col" + name])
        if via == "delay":
            d["delay" + name] = torch.randint(1, 51, (m,), generator=gen, device=_device(), dtype=torch.uint8)
        elif via == "synapses":
            d["w" + name] = torch.rand(m, generator=gen, device=_device(), dtype=torch.float64) + 0.5
            d["delay" + name] = torch.randint(0, 40, (m,), generator=gen, device=_device(), dtype=torch.uint8)
    d["v0"] = VR + torch.rand(n, generator=gen, device=_device(), dtype=torch.float64) * (VT - VR)
    return d


def _weights(c):
    """Excitatory and inhibitory weight: the reference's for 80 synapses per
    neuron, scaled with the in-degree (delayed networks as the benchmark's:
    0.162 and -0.9 mV for 1000)."""
    s = (100.0 if c.get("via") == "delay" else 80.0) / c["indegree"]
    return 1.62 * mV * s, -9 * mV * s


def _cuba_eqs():
    return b.Equations("""
    dv/dt  = (ge+gi-(v-El))/taum : volt
    dge/dt = -ge/taue : volt
    dgi/dt = -gi/taui : volt
    """, taum=TAUM, taue=TAUE, taui=TAUI, El=EL)


def _host(x):
    return x.cpu().numpy()


def _network(c, seed):
    d = _wiring(c, seed)
    n, ne, via = d["n"], d["ne"], c.get("via", "connection")
    clock = b.Clock(dt=DT)
    if c["kind"] == "coba":
        eqs = b.Equations("""
        dv/dt  = (ge*(Ee-v) + gi*(Ei-v) + (El-v))/taum : volt
        dge/dt = -ge/taue : 1
        dgi/dt = -gi/taui : 1
        """, taum=TAUM, taue=TAUE, taui=TAUI, Ee=EE, Ei=EI, El=EL)
        P = b.NeuronGroup(n, model=eqs, threshold=VT, reset=VR, clock=clock, method=c["method"])
        we, wi = 0.027 * 80.0 / c["indegree"], 0.18 * 80.0 / c["indegree"]
    else:
        P = b.NeuronGroup(n, model=_cuba_eqs(), threshold=VT, reset=VR, clock=clock)
        we, wi = _weights(c)
    Pe, Pi = P.subgroup(ne), P.subgroup(n - ne)
    objs = [P]
    for name, src, var, w in (("e", Pe, "ge", we), ("i", Pi, "gi", wi)):
        row, col = _host(d["row" + name]), _host(d["col" + name])
        if via == "synapses":
            S = b.Synapses(src, P, model="w : volt", pre="%s += w" % var, clock=clock)
            S.create_synapses(np.repeat(np.arange(len(src)), np.diff(row)), col)
            S.w = w * _host(d["w" + name])
            S.delay = (_host(d["delay" + name]) + 0.5) * DT
            objs.append(S)
        elif via == "delay":
            C = b.DelayConnection(src, P, var, max_delay=5 * ms, dtype=np.float32)
            C.connect_csr(row, col, np.float32(w), delay_steps=_host(d["delay" + name]))
            objs.append(C)
        else:
            C = b.Connection(src, P, var)
            C.connect_csr(row, col, w)
            objs.append(C)
    P.v = _host(d["v0"])
    M = b.SpikeMonitor(P)
    return dict(net=b.Network(*(objs + [M])), P=P, M=M)


def _room(n, c):
    """Length of a spike record's arrays, above the spikes expected
    (a record is padded to it with -1, so that its shape does not depend on
    the seed)."""
    hz = {"net": 4.0 if c.get("via") == "delay" else 10.0, "coba": 20.0, "batch": 10.0, "stdp": 6000.0}[c["kind"]]
    return int(n * c["steps"] * DT * hz) + n // 8


def _padded(i, t, room):
    oi, ot = np.full(room, -1, dtype=np.int32), np.full(room, -1.0)
    k = min(len(i), room)
    oi[:k], ot[:k] = i[:k], t[:k]
    return oi, ot


def _read(s, c):
    out = {}
    i, t = s["M"].it
    s["M"].reinit()                      # the records are read: the next run's start empty
    out["i"], out["t"] = _padded(i, t, _room(len(s["P"]), c))
    for v in s["P"]._names:
        out[v] = np.array(getattr(s["P"], v))
    return out


def _build_net(c, seed):
    b.set_global_preferences(precision=c.get("precision", 64))
    try:
        s = _network(c, seed)
        s["net"].prepare()
    finally:
        b.set_global_preferences(precision=64)
    return s


def _build_batch(c, seed):
    parts = [_network(dict(c, kind="net"), seed * 1009 + r) for r in range(c["count"])]
    batch = b.NetworkBatch([p["net"] for p in parts])
    for p in parts:
        p["net"].prepare()
    return dict(batch=batch, parts=parts)


def _build_stdp(c, seed):
    clock = b.Clock(dt=DT)
    gen = _generator(seed)
    nin, nout, gmax = c["nin"], c["nout"], 0.01
    eqs = b.Equations("""
    dv/dt=(ge*(Ee-vr)+El-v)/taum : volt
    dge/dt=-ge/taue : 1
    """, taum=10 * ms, taue=5 * ms, Ee=0 * mV, vr=-60 * mV, El=-74 * mV)
    rates = _host(5.0 + 20.0 * torch.rand(nin, generator=gen, device=_device(), dtype=torch.float64))
    inputs = b.PoissonGroup(nin, rates=rates * Hz, clock=clock, seed=seed + 1)
    outputs = b.NeuronGroup(nout, model=eqs, threshold=-54 * mV, reset=-60 * mV, clock=clock)
    outputs.v = -60 * mV
    C = b.Connection(inputs, outputs, "ge", structure="dense", dtype=np.float32)
    C.connect(W=_host(gmax * torch.rand((nin, nout), generator=gen, device=_device(), dtype=torch.float64)))
    stdp = b.ExponentialSTDP(C, 20 * ms, 20 * ms, 0.01, -0.0105, wmax=gmax)
    M = b.SpikeMonitor(outputs.subgroup(min(64, nout)))
    net = b.Network(inputs, outputs, C, stdp, M)
    net.prepare()
    return dict(net=net, outputs=outputs, C=C, stdp=stdp, M=M)


def _run_stdp(c, s):
    s["net"].run(c["steps"] * DT)
    i, t = s["M"].it
    s["M"].reinit()
    i, t = _padded(i, t, _room(len(s["M"].source), c))
    pre, post = s["stdp"]._traces()
    return {"i": i, "t": t, "w": s["C"]._weights(), "v": np.array(s["outputs"].v), "ge": np.array(s["outputs"].ge),
            "pre": np.array(pre), "post": np.array(post)}


# ----------------------------------------------------------------- fitting
def _fit_data(c, seed):
    w = FitWorkload(ntargets=c["targets"], dur_min=min(1.0, c["seconds"]), dur_max=c["seconds"], dt=DT, seed=seed)
    w.build_targets()
    return w


def _candidates(n, seed):
    rng = np.random.default_rng(seed)
    return np.array([np.exp(np.log(lo) + (np.log(hi) - np.log(lo)) * rng.random(n))
                     for lo, hi in (PRIOR[k] for k in PARAMS)])


def _build_fit(c, seed):
    w = _fit_data(c, seed)
    prob = FittingProblem(adaptive_lif_equations(), THRESHOLD, RESET, w.targets, w.inputs, DT, c["particles"],
                          precision=c["precision"], method=c["method"], param_names=list(PARAMS))
    return dict(prob=prob, X=_candidates(prob.N, seed + 1))


def _build_fitcall(c, seed):
    w = _fit_data(c, seed)
    box = {k: [PRIOR[k][0] / 2, PRIOR[k][1] * 2] for k in PARAMS}
    return dict(data=w.data(), inputs=w.inputs, box=box, seed=seed % 100003)


def _run_fitcall(c, s):
    r = modelfitting(model=adaptive_lif_equations(), reset=RESET, threshold=THRESHOLD, data=s["data"],
                     input=s["inputs"], dt=DT, popsize=c["particles"], maxiter=c["iterations"], delta=4 * ms,
                     precision=c["precision"], method=c["method"], algorithm=PSO, seed=s["seed"], **s["box"])
    pos = r.best_pos if isinstance(r.best_pos, list) else [r.best_pos]
    return {"fit": np.atleast_1d(np.asarray(r.best_fit, dtype=np.float64)),
            "pos": np.array([[p[k] for k in PARAMS] for p in pos]), "trace": r.info["trace"]}


# -------------------------------------------------------- proposal network
def _mlp_data(rows, seed):
    """Parameters of the network's shape (He-style, small output layer), and
    normalised features with targets in [-1, 1]."""
    gen = _generator(seed)
    params = []
    for l in range(4):
        W = torch.randn((MLP_ROWS[l], MLP_COLS[l]), generator=gen, device=_device()) * math.sqrt(2.0 / MLP_COLS[l])
        bias = 0.02 * torch.randn(MLP_ROWS[l], generator=gen, device=_device())
        if l == 3:
            W *= 0.05
            W[2 * YDIM:] = 0
            bias[2 * YDIM:] = 0
        params.append((W, bias))
    X = torch.randn((rows, 64), generator=gen, device=_device())
    mix = torch.randn((64, YDIM), generator=gen, device=_device()) / 8.0
    Y = torch.tanh(X @ mix + 0.3 * torch.randn((rows, YDIM), generator=gen, device=_device()))
    return params, X, Y


def _build_mlp(c, seed):
    rows = c.get("rows", c["batch"])
    params, X, Y = _mlp_data(rows, seed)
    h = MLPHandle(YDIM)
    for l, (W, bias) in enumerate(params):
        h.set_params(l, _host(W), _host(bias))
    h.set_data(_host(X), _host(Y))
    if c["kind"] == "grad":
        h.epoch_order(seed, 0)
    return dict(h=h, seed=seed % 100003)


def _run_train(c, s):
    loss, _ = s["h"].train(c["epochs"], c["batch"], 1e-3, s["seed"])
    out = {"loss": loss}
    for l in range(4):
        out["W%d" % l], out["b%d" % l] = s["h"].get_params(l)
    return out


def _run_grad(c, s):
    loss, g = s["h"].step_gradients(c["batch"], 0)
    # the vector lives in the handle: what is kept beyond it is a copy
    return {"loss": np.float32(loss), "grad": g.torch().clone()}


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("net", "coba"):
        s = _build_net(c, seed)
    elif kind == "batch":
        s = _build_batch(c, seed)
    elif kind == "stdp":
        s = _build_stdp(c, seed)
    elif kind == "fit":
        s = _build_fit(c, seed)
    elif kind == "fitcall":
        s = _build_fitcall(c, seed)
    else:
        s = _build_mlp(c, seed)
    s["case"] = c
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("net", "coba"):
        state["net"].run(c["steps"] * DT)
        return _read(state, c)
    if kind == "batch":
        state["batch"].run(c["steps"] * DT)
        # one array per quantity over all networks
        parts = [_read(p, c) for p in state["parts"]]
        return {k: np.concatenate([p[k] for p in parts]) for k in ("i", "t", "v", "ge", "gi")}
    if kind == "stdp":
        return _run_stdp(c, state)
    if kind == "fit":
        return state["prob"].evaluate(state["X"])
    if kind == "fitcall":
        return _run_fitcall(c, state)
    if kind == "grad":
        return _run_grad(c, state)
    return _run_train(c, state)


# -------------------------------------------------------------------- work
def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind in ("net", "coba", "batch"):
        nets, n, steps = c.get("count", 1), c["n"], c["steps"]
        size = c.get("precision", 64) // 8
        # about 10 spikes per neuron and second; a spike's row is read (target, and weight or delay where it has its own)
        events = 10.0 * n * steps * DT * c["indegree"] * nets
        per = {"connection": 4, "delay": 5, "synapses": 13}[c.get("via", "connection")]
        state = nets * n * 3 * size
        records = 10.0 * n * steps * DT * 12 * nets
        return {"bytes": 2 * state + nets * n * 24 + events * per + records,
                "flops": nets * n * steps * (14.0 if kind == "coba" else 11.0) + events}
    if kind == "stdp":
        nin, nout, steps = c["nin"], c["nout"], c["steps"]
        pre = 15.0 * nin * steps * DT * nout                 # weights touched by input spikes
        # outputs of few inputs hardly fire; of many they fire on about half the steps
        post = min(0.5, nin / 20000.0) * nout * steps * nin
        return {"bytes": nin * nout * 12.0 + (nin + nout) * 32.0, "flops": 3 * pre + 3 * post + 8.0 * nout * steps}
    if kind in ("fit", "fitcall"):
        size = 4 if c["precision"] == "float" else 8
        mean_s = (min(1.0, c["seconds"]) + c["seconds"]) / 2
        steps = c["targets"] * mean_s / DT
        evaluations = c.get("iterations", 0) + 1
        sims = c["targets"] * c["particles"]
        per = {"Euler": 10.0, "RK": 22.0, "exponential_Euler": 40.0}[c["method"]]
        return {"bytes": evaluations * (steps * size + sims * (len(PARAMS) * 8 + 8)),
                "flops": evaluations * steps * c["particles"] * per}
    weights = sum(r * k for r, k in zip(MLP_ROWS, MLP_COLS))
    batch = c["batch"]
    steps = 1 if kind == "grad" else c["epochs"] * (c["rows"] // batch)
    flops = batch * (3 * 2 * weights - 2 * 64 * 512) * float(steps)
    moved = batch * (64 + YDIM) * 4.0 * steps + weights * (8.0 if kind == "grad" else 4.0 * 6)
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------- exact
def _exact_net(wires, c):
    """The networks of `wires` (independent of one another) as one, in 64-bit
    torch: the linear update by the matrix exponential or the scheme of the
    nonlinear model, threshold, arrivals due, reset."""
    dev = _device()
    coba = c["kind"] == "coba"
    via = c.get("via", "connection")
    steps, n = c["steps"], wires[0]["n"]
    total = n * len(wires)
    dt = DT
    if coba:
        we, wi = 0.027 * 80.0 / c["indegree"], 0.18 * 80.0 / c["indegree"]
    else:
        we, wi = _weights(c)
    if via == "delay":
        we, wi = float(np.float32(we)), float(np.float32(wi))
    deg = torch.zeros(total, dtype=torch.int64, device=dev)
    cols, wts, dly, exc = [], [], [], []
    for r, d in enumerate(wires):
        for name, w in (("e", we), ("i", wi)):
            m = len(d["col" + name])
            cols.append(d["col" + name].to(torch.int64) + r * n)
            wts.append(d["w" + name] * w if via == "synapses" else torch.full((m,), w, dtype=torch.float64, device=dev))
            dly.append(d["delay" + name] if "delay" + name in d else torch.zeros(m, dtype=torch.uint8, device=dev))
            lo = r * n + (0 if name == "e" else d["ne"])
            deg[lo:lo + len(d["row" + name]) - 1] = torch.diff(d["row" + name])
        exc.append(torch.arange(n, device=dev) < d["ne"])
    cols, wts, dly, exc = torch.cat(cols), torch.cat(wts), torch.cat(dly), torch.cat(exc)
    start = torch.zeros(total + 1, dtype=torch.int64, device=dev)
    torch.cumsum(deg, 0, out=start[1:])
    depth = 51 if via != "connection" else 1
    ring = torch.zeros((depth, 2 * total), dtype=torch.float64, device=dev)
    flat = ring.reshape(-1)
    v = torch.cat([d["v0"] for d in wires])
    ge, gi = torch.zeros_like(v), torch.zeros_like(v)
    A = torch.zeros((3, 3), dtype=torch.float64)
    A[0] = torch.tensor([-1 / TAUM, 1 / TAUM, 1 / TAUM])
    A[1, 1], A[2, 2] = -1 / TAUE, -1 / TAUI
    E = torch.matrix_exp(A * dt)
    E00, E01, E02, E11, E22 = (float(E[i, j]) for i, j in ((0, 0), (0, 1), (0, 2), (1, 1), (2, 2)))
    shift = EL - E00 * EL

    def rhs(v, ge, gi):
        return (ge * (EE - v) + gi * (EI - v) + (EL - v)) / TAUM, -ge / TAUE, -gi / TAUI

    si, st = [], []
    for t in range(steps):
        if not coba:
            v = E00 * v + E01 * ge + E02 * gi + shift
            ge, gi = E11 * ge, E22 * gi
        elif c["method"] == "Euler":
            dv, de, di = rhs(v, ge, gi)
            v, ge, gi = v + dt * dv, ge + dt * de, gi + dt * di
        elif c["method"] == "RK":
            dv, de, di = rhs(v, ge, gi)
            dv, de, di = rhs(v + 0.5 * dt * dv, ge + 0.5 * dt * de, gi + 0.5 * dt * di)
            v, ge, gi = v + dt * dv, ge + dt * de, gi + dt * di
        else:
            # dx/dt = a x + b at the step's start: x <- (x + b/a) exp(a dt) - b/a
            b0 = (ge * EE + gi * EI + EL) / TAUM
            a0 = ((ge * (EE - 1) + gi * (EI - 1) + (EL - 1)) / TAUM) - b0
            q = b0 / a0
            v = (v + q) * torch.exp(a0 * dt) - q
            ge, gi = ge * math.exp(-dt / TAUE), gi * math.exp(-dt / TAUI)
        spk = torch.nonzero(v > VT).reshape(-1)
        if len(spk):
            cnt = deg[spk]
            pos = torch.repeat_interleave(start[spk] - torch.cumsum(cnt, 0) + cnt, cnt) + torch.arange(
                int(cnt.sum()), device=dev)
            side = torch.where(torch.repeat_interleave(exc[spk], cnt), 0, total)
            row = (t + dly[pos].to(torch.int64)) % depth
            flat.index_add_(0, row * (2 * total) + side + cols[pos], wts[pos])
        due = ring[t % depth]
        ge, gi = ge + due[:total], gi + due[total:]
        due.zero_()
        v[spk] = VR
        si.append(spk)
        st.append(torch.full((len(spk),), t, dtype=torch.int64, device=dev))
    si, st = torch.cat(si), torch.cat(st)
    si, st = _host(si), _host(st) * dt
    net = si // n
    rec = [_padded(si[net == r] - r * n, st[net == r], _room(n, c)) for r in range(len(wires))]
    return {"i": np.concatenate([r[0] for r in rec]), "t": np.concatenate([r[1] for r in rec]),
            "v": v, "ge": ge, "gi": gi}


def _exact_gamma(c, seed):
    """Gamma of every candidate: the model's steps in 64-bit torch, then the
    exclusive coincidence count spike by spike."""
    w = _fit_data(c, seed)
    if c["precision"] != "double" or c["method"] != "Euler":
        return None
    pop, delta = c["particles"], 40
    X = _candidates(c["targets"] * pop, seed + 1)
    if max(len(x) for x in w.inputs) > 40000 or X.shape[1] > 4096:
        return None
    dev = _device()
    out = np.empty(X.shape[1])
    for j, (inp, tgt) in enumerate(zip(w.inputs, w.targets)):
        R, tau, Vt0, alpha, tau_t = (torch.from_numpy(X[d, j * pop:(j + 1) * pop].copy()).to(dev) for d in range(5))
        L = int((len(inp) * DT) / DT)
        V, Vt = torch.zeros(pop, dtype=torch.float64, device=dev), torch.zeros(pop, dtype=torch.float64, device=dev)
        raster = torch.zeros((L, pop), dtype=torch.bool, device=dev)
        for T in range(L):
            dV, dVt = (R * float(inp[T]) - V) / tau, (Vt0 - Vt) / tau_t
            V, Vt = V + dV * DT, Vt + dVt * DT
            s = V > Vt
            raster[T] = s
            V = torch.where(s, 0.0, V)
            Vt = torch.where(s, Vt + alpha, Vt)
        raster = raster.cpu().numpy()
        steps = np.rint(np.hstack(([-1.0], np.sort(tgt), [len(inp) * DT + 1.0])) / DT).astype(np.int64)
        rate = (len(tgt) - 1) / (max(tgt) - min(tgt)) if len(tgt) > 1 else np.nan
        for k in range(pop):
            spikes = np.nonzero(raster[:, k])[0]
            at, last_ok, next_ok, hits = 0, False, True, 0
            for T in spikes:
                while at + 1 < len(steps) and steps[at + 1] < T:       # the train's position moves past earlier steps
                    at += 1
                    last_ok, next_ok = next_ok, True
                nxt = steps[at + 1] if at + 1 < len(steps) else 2 ** 31 - 1
                near_last, near_next = steps[at] + delta >= T, nxt - delta <= T
                ml, mn = near_last and last_ok, near_next and next_ok
                hits += bool(ml or mn)
                last_ok = last_ok and not near_last
                next_ok = (next_ok and not near_next) or (ml and mn)
            avg = 2 * 4e-3 * len(tgt) * rate
            norm = .5 * (1 - 2 * 4e-3 * rate)
            with np.errstate(divide="ignore", invalid="ignore"):
                out[j * pop + k] = np.float64(hits - avg) / (norm * (len(tgt) + len(spikes)))
    return out


def _exact_grad(c, seed):
    """Loss and gradient in 64-bit torch (no rounding of the activations):
    one batch holds the whole training set, so the row order only permutes
    the sum."""
    params, X, Y = _mlp_data(c["batch"], seed)
    P = [(W.double().requires_grad_(), bias.double().requires_grad_()) for W, bias in params]
    h = X.double()
    for l in range(3):
        h = torch.relu(h @ P[l][0].t() + P[l][1])
    o = h @ P[3][0].t() + P[3][1]
    mu, sr = o[:, :YDIM], o[:, YDIM:2 * YDIM]
    s = torch.clamp(sr, -7.0, 7.0)
    r = (Y.double() - mu) * torch.exp(-s)
    loss = (0.5 * r * r + s).sum() / len(X)
    loss.backward()
    flat = torch.cat([g.grad.reshape(-1) for pair in P for g in pair])
    return {"loss": float(loss), "grad": flat}


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "net" and c.get("precision", 64) == 32:
        return None                        # its spikes leave the 64-bit ones after a few steps
    if kind in ("net", "coba"):
        if c["steps"] * c["n"] * c["indegree"] > 6e11:
            return None
        return _exact_net([_wiring(c, seed)], c)
    if kind == "batch":
        return _exact_net([_wiring(c, seed * 1009 + r) for r in range(c["count"])], c)
    if kind == "fit":
        return _exact_gamma(c, seed)
    if kind == "grad":
        return _exact_grad(c, seed)
    return None                            # long plastic or training runs: no such value
