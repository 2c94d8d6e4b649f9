"""Networks on a device without room for what a persistent launch or pending
STDP updates keep besides the network itself: smaller bins, else the stepped
launches or every step's updates, with the oracle's results and the buffers
that were not used given back."""
import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import Hz, ms, mV
from brian_b200._lib import EngineError
from brian_b200.network import engine

pytestmark = pytest.mark.gpu

BG_ENOMEM = -2


def _synapses():
    rng = np.random.default_rng(1)
    P = b.NeuronGroup(3000, model="dv/dt = (20*mV - v)/(10*ms) : volt", threshold=10 * mV, reset=0 * mV)
    P.v = rng.random(3000) * 10 * mV
    S = b.Synapses(P, P, model="w : volt", pre="v += w")
    S.create_synapses(np.repeat(np.arange(3000), 20), np.concatenate([np.sort(rng.choice(3000, 20, replace=False)) for _ in range(3000)]))
    S.w = rng.random(60000) * 0.1 * mV
    S.delay = rng.random(60000) * 3 * ms
    return [P, S], P


def _direct(method="linear"):
    rng = np.random.default_rng(2)
    P = b.NeuronGroup(3000, model="dv/dt = (20*mV - v)/(10*ms) : volt", threshold=10 * mV, reset=0 * mV,
                      **({} if method == "linear" else dict(method=method)))
    P.v = rng.random(3000) * 10 * mV
    C = b.Connection(P, P, "v")
    C.connect_csr(np.arange(3001, dtype=np.int64) * 20,
                  np.concatenate([np.sort(rng.choice(3000, 20, replace=False)) for _ in range(3000)]).astype(np.int32), 0.1 * mV)
    return [P, C], P


def _generated():
    return _direct("Euler")


def _stdp():
    rng = np.random.default_rng(3)
    src = b.PoissonGroup(2000, rates=30 * Hz, seed=5)
    P = b.NeuronGroup(50, model="dv/dt = (ge - v)/(10*ms) : volt\ndge/dt = -ge/(5*ms) : volt", threshold=10 * mV, reset=0 * mV)
    C = b.Connection(src, P, "ge", structure="dense", dtype=np.float32)
    C.connect(W=rng.random((2000, 50)) * 4e-3)
    return [src, P, C, b.ExponentialSTDP(C, 20 * ms, 20 * ms, 0.01, -0.0105, wmax=4e-3)], P


def _run(build, limit=0):
    b.clear()
    b.reinit_default_clock()
    objs, P = build()
    M = b.SpikeMonitor(P)
    net = b.Network(*(objs + [M]))
    net.prepare(configure=(lambda rt: rt.debug_device_limit(limit)) if limit else None)
    held = net.stats().get("device_bytes")
    for _ in range(2):
        net.run(10 * ms)
    out = scenarios._result(net, groups=[P], spikemons=[M])
    if build is _stdp:
        out["W"] = objs[2]._weights().astype(np.float64)
    th = net.stats().get("persistent_threads")
    net._invalidate()
    return out, held, th


# bytes that the network runs without at least; whether it runs persistent with all of them
@pytest.mark.parametrize("build,part,persistent", [(_synapses, 8, True), (_direct, 64, True), (_generated, 64, True), (_stdp, 800, False)])
def test_less_and_less_memory(oracle_table, gpu_table, build, part, persistent):
    with engine(oracle_table):
        ref = _run(build)[0]
    gpu, full, th = _run(build)
    scenarios.compare(ref, gpu)
    assert (th > 0) == persistent and len(ref["spk0.idx"]) > 50
    ran, stepped, held = 0, 0, []
    for limit in [full - int(1.3 ** k) for k in range(0, 90, 4) if 1.3 ** k < full]:
        try:
            gpu, used, th = _run(build, limit)
        except EngineError as e:
            assert e.code == BG_ENOMEM, e            # not even the network itself
            break
        scenarios.compare(ref, gpu)
        assert used <= limit
        ran += 1
        stepped += th == 0
        held.append(used)
    assert ran >= 1 and stepped >= 1 and min(held) <= full - part
    if build is _synapses:
        assert stepped < ran                         # with smaller bins first
