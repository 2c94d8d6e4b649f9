"""Pushes of the persistent kernel (networks past the cluster kernel's size):
rows of synapses at the edges of what a warp and its four loads cover, empty
rows, sources in both connections, steps in which every neuron of a block
spikes, zero and longer delays; states and spikes equal the oracle's."""
import numpy as np
import pytest

import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu


def _run(n, lens, drive, delayed):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(n)
    P = b.NeuronGroup(n, model="dv/dt = (ge + gi - v + %g*mV)/(10*ms) : volt\ndge/dt = -ge/(5*ms) : volt\ndgi/dt = -gi/(10*ms) : volt"
                      % drive, threshold=10 * mV, reset=0 * mV)
    P.v = rng.random(n) * 10 * mV
    conns = []
    for src, var, w in ((P, "ge", 0.02 * mV), (P[n // 2:], "gi", -0.03 * mV)):
        m = len(src)
        row = np.zeros(m + 1, dtype=np.int64)
        row[1:] = np.cumsum(np.asarray(lens)[np.arange(m) % len(lens)])
        cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in np.diff(row)] or [np.zeros(0)]).astype(np.int32)
        if delayed:
            C = b.DelayConnection(src, P, var, max_delay=2 * ms)
            C.connect_csr(row, cols, w, delay_steps=rng.integers(1, 21, len(cols)).astype(np.uint8))
        else:
            C = b.Connection(src, P, var)
            C.connect_csr(row, cols, w)
        conns.append(C)
    M = b.SpikeMonitor(P)
    net = b.Network(P, M, *conns)
    net.run(3 * ms)
    net.run(0.7 * ms)
    s, i = M._record()
    return s.copy(), i.copy(), np.array(P.v), np.array(P.ge), np.array(P.gi), net.stats().get("persistent_threads", 0)


@pytest.mark.parametrize("n,lens,drive,delayed", [
    (20011, (0, 1, 31, 32, 33), 14, True),                 # one warp a row
    (20011, (127, 128, 129, 0, 300), 14, True),            # two
    (18433, (0, 0, 0, 2600, 1), 14, True),                 # four, uneven rows
    (17000, (1100,), 14, False),
    (18433, (3, 0, 5), 4000, True),                        # every neuron in the same step
])
def test_push(oracle_table, gpu_table, n, lens, drive, delayed):
    out = []
    for tab in (oracle_table, gpu_table):
        with engine(tab):
            out.append(_run(n, lens, drive, delayed))
    ref, got = out
    assert got[5] > 0 and len(ref[0]) > 0
    for x, y in zip(ref[:5], got[:5]):
        assert np.array_equal(x, y)
