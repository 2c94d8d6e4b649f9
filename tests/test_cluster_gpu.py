"""Small networks in the cluster kernel (one block, or a thread-block cluster)
against the oracle, bit for bit (FP64; FP32 against the engine's persistent
kernel, whose arithmetic it shares): sizes at the edges of the blocks and of
the neurons per thread, every pattern of delivered variables, zero and longer
delays, subgroups, bursts in which every neuron spikes at once, StateMonitors
with repeated neurons and periods, split runs, generated models."""
import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu

EQS = {
    # delivered variables, equations
    "up": (("ge", "gi"), "dv/dt = (ge+gi-(v-El))/taum : volt\ndge/dt = -ge/taue : volt\ndgi/dt = -gi/taui : volt"),
    "swapped": (("gi", "ge"), "dv/dt = (ge+gi-(v-El))/taum : volt\ndge/dt = -ge/taue : volt\ndgi/dt = -gi/taui : volt"),
    "same": (("ge", "ge"), "dv/dt = (ge-(v-El))/taum : volt\ndge/dt = -ge/taue : volt"),
    "delta": (("v", "v"), "dv/dt = -(v-El)/taum : volt"),
    "delta2": (("v", "v"), "dv/dt = (ge-(v-El))/taum : volt\ndge/dt = -ge/taue : volt"),
    "last": (("x", "x"), "dx/dt = -x/taue : volt\ndv/dt = (x-(v-El))/taum : volt"),
    "four": (("ge", "gi"), "dv/dt = (ge+gi-w-(v-El))/taum : volt\ndge/dt = -ge/taue : volt\ndgi/dt = -gi/taui : volt\n"
                          "dw/dt = (0.1*(v-El)-w)/taui : volt"),
}
CONST = dict(taum=20 * ms, taue=5 * ms, taui=10 * ms, El=-49 * mV)


def _csr(rng, n_src, n_tgt, k):
    """About k targets per source, ascending; some sources without any."""
    rows = [np.sort(rng.choice(n_tgt, min(n_tgt, int(c)), replace=False)) for c in rng.integers(0, 2 * k + 1, n_src)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return ptr, (np.concatenate(rows) if len(rows) else np.zeros(0)).astype(np.int32)


def _run(n, eqs="up", kind="connection", steps=120, k=12, burst=False, dmin=1, runs=2, model=None, sub=False,
         record=None, timestep=1, seed=5):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(seed + n)
    kw = dict(threshold=-50 * mV, reset=-60 * mV)
    if model is not None:
        kw.update(model)
    P = b.NeuronGroup(n, model=b.Equations(EQS[eqs][1], **CONST), **kw)
    ne = max(1, int(0.8 * n)) if n > 1 else 1
    parts = [P.subgroup(ne)] + ([P.subgroup(n - ne)] if n > ne else [])
    target = P[n // 3:n] if sub and n > 3 else P
    conns = []
    for i, src in enumerate(parts):
        var, w = EQS[eqs][0][i], (1.1 * mV, -2.3 * mV)[i]
        ptr, cols = _csr(rng, len(src), len(target), k)
        if kind == "delay" or (kind == "mixed" and i == 1):
            C = b.DelayConnection(src, target, var, max_delay=3 * ms)
            C.connect_csr(ptr, cols, w, delay_steps=rng.integers(dmin, 31, len(cols)).astype(np.uint8))
        else:
            C = b.Connection(src, target, var)
            C.connect_csr(ptr, cols, w)
        conns.append(C)
    P.v = -40 * mV if burst else -60 * mV + rng.random(n) * 14 * mV
    M = b.SpikeMonitor(P)
    mons = [M, b.SpikeMonitor(parts[0])]
    S = b.StateMonitor(P, "v", record=[i for i in (record or [0, n - 1, n // 2, 0]) if i < n], timestep=timestep)
    net = b.Network(P, *(conns + mons + [S]))
    for _ in range(runs):
        net.run(steps * 0.1 * ms)
    out = scenarios._result(net, groups=[P], spikemons=mons, statemons=[S])
    th = net.stats().get("persistent_threads", 0)
    net._invalidate()
    return out, th


def _both(oracle_table, **kw):
    with engine(oracle_table):
        ref, _ = _run(**kw)
    gpu, th = _run(**kw)
    assert th == 512
    scenarios.compare(ref, gpu)
    return ref


@pytest.mark.parametrize("n", [1, 31, 512, 513, 1024, 1025, 2047, 2048, 2049, 4097, 8192, 8193, 20000])
@pytest.mark.parametrize("kind", ["connection", "delay"])
def test_sizes(oracle_table, gpu_table, n, kind):
    r = _both(oracle_table, n=n, kind=kind, steps=60 if n > 5000 else 120)
    assert n < 100 or len(r["spk0.idx"]) > 0


@pytest.mark.parametrize("eqs", sorted(EQS))
@pytest.mark.parametrize("n,kind,dmin", [(700, "connection", 1), (3000, "connection", 1), (700, "delay", 0),
                                         (3000, "delay", 0), (3000, "delay", 1), (3000, "mixed", 1)])
def test_patterns(oracle_table, gpu_table, eqs, n, kind, dmin):
    _both(oracle_table, n=n, eqs=eqs, kind=kind, dmin=dmin, sub=True, record=[n - 1, 5, 5, n // 2], timestep=3)


@pytest.mark.parametrize("n,kind", [(900, "connection"), (5000, "connection"), (5000, "delay"), (5000, "mixed")])
def test_burst(oracle_table, gpu_table, n, kind):
    """Every neuron spikes in the first step: many events per target and step."""
    _both(oracle_table, n=n, kind=kind, burst=True, k=30, steps=40)


@pytest.mark.parametrize("n", [600, 3000])
@pytest.mark.parametrize("model", [dict(threshold="v > -50*mV + 1*mV*(t > 5*ms)", reset="v = -60*mV\nge *= 0.5"),
                                   dict(method="Euler"), dict(method="RK"),
                                   dict(method="Euler", threshold="v > -50*mV", reset=-60 * mV)])
def test_generated(oracle_table, gpu_table, n, model):
    _both(oracle_table, n=n, model=model, kind="mixed")


@pytest.mark.parametrize("kind", ["connection", "delay"])
@pytest.mark.parametrize("n", [1500, 6000])
def test_fp32_equals_persistent_kernel(gpu_table, n, kind):
    outs = []
    b.set_global_preferences(precision=32)
    try:
        for p in (True, 512):
            b.set_global_preferences(persistent=p)
            outs.append(_run(n=n, kind=kind)[0])
    finally:
        b.set_global_preferences(precision=64, persistent=True)
    scenarios.compare(outs[0], outs[1])


def test_wide_rows_take_the_persistent_kernel(oracle_table, gpu_table):
    """More synapses into a block than its transaction count holds."""
    _both(oracle_table, n=3000, kind="connection", k=700, steps=20)


def test_networks_side_by_side(oracle_table, gpu_table):
    """Networks of different sizes prepared together run by turns: the launch
    limits of one do not depend on another's."""
    refs, nets = [], []
    for n, k in ((3000, 60), (1500, 10), (6000, 30)):
        for tab in (oracle_table, None):
            P = b.NeuronGroup(n, model=b.Equations(EQS["up"][1], **CONST), threshold=-50 * mV, reset=-60 * mV,
                              clock=b.Clock(dt=0.1 * ms))
            rng = np.random.default_rng(n)
            C = b.Connection(P, P, "ge")
            C.connect_csr(*_csr(rng, n, n, k), 0.8 * mV)
            P.v = -60 * mV + rng.random(n) * 14 * mV
            net = b.Network(P, C)
            if tab is None:
                net.prepare()
            else:
                with engine(tab):
                    net.prepare()
            (nets if tab is None else refs).append((net, P))
    for _ in range(2):
        for (net, P), (ref, Q) in zip(nets, refs):
            net.run(5 * ms)
            ref.run(5 * ms)
    for (net, P), (ref, Q) in zip(nets, refs):
        assert net.stats()["persistent_threads"] == 512
        for v in ("v", "ge", "gi"):
            assert np.array_equal(np.asarray(getattr(P, v)), np.asarray(getattr(Q, v)))
        net._invalidate()
        ref._invalidate()
