"""The persistent kernel for Synapses keeps events on their way in a ring of
bins: the oracle's spikes and states, bit for bit, with no delay, one delay, the
longest, several of a target in one step (up to and past the number it orders
without a sort), bins at the edges of the group, more sources in one step than
a block has warps, split runs, runs shorter than the delays, and weights
changed while events are on their way."""
import numpy as np
import pytest

import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu


def _run(n, delay, k, runs, subgroups, change, drive):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(n + k)
    G = b.NeuronGroup(n, model="dv/dt = (ge - v + %g*mV)/(10*ms) : volt\ndge/dt = -ge/(5*ms) : volt" % drive, threshold=10 * mV,
                      reset=0 * mV)
    G.v = rng.random(n) * 10 * mV
    parts = [(G[:n // 3], "ge += w"), (G[n // 3:], "v -= w")] if subgroups else [(G, "ge += w")]
    objs = []
    for src, code in parts:
        S = b.Synapses(src, G, model="w : volt", pre=code)
        S.connect_random(sparseness=min(1.0, 4.0 * k / n))
        S.w = "0.05*mV * (1 + ((3*i + 7*j) % 11))"
        S.delay = delay
        objs.append(S)
    M = b.SpikeMonitor(G)
    net = b.Network(G, M, *objs)
    for r, steps in enumerate(runs):
        if change and r:
            for S in objs:
                S.w = "0.03*mV * (1 + ((5*i + j) %% %d))" % (7 + r)
        net.run(steps * 0.1 * ms)
    s, i = M._record()
    return s.copy(), i.copy(), np.array(G.v), np.array(G.ge), net.stats().get("persistent_threads", 0)


@pytest.mark.parametrize("n,delay,k,runs,subgroups,change,drive", [
    (1, "0*ms", 1, (40,), False, False, 30),
    (1023, "0*ms", 1, (60,), False, False, 14),
    (1025, "0.1*ms", 2, (60, 1, 1, 40), True, False, 14),
    (2049, "rand() * 3*ms", 1, (50, 7, 30), True, False, 14),
    (2049, "rand() * 3*ms", 1, (50, 7, 30), True, True, 14),
    (1500, "25.4*ms", 1, (100, 200, 100), False, True, 14),
    (600, "rand() * 0.3*ms", 6, (80,), True, False, 60),      # many spikes a step, many events a target
])
def test_ring(oracle_table, gpu_table, n, delay, k, runs, subgroups, change, drive):
    b.set_global_preferences(synapse_events=True)
    try:
        out = []
        for tab in (oracle_table, gpu_table):
            np.random.seed(11)
            with engine(tab):
                out.append(_run(n, delay, k, runs, subgroups, change, drive))
    finally:
        b.set_global_preferences(synapse_events=None)
    ref, got = out
    assert got[4] > 0 and len(ref[0]) > 0
    for x, y in zip(ref[:4], got[:4]):
        assert np.array_equal(x, y)
