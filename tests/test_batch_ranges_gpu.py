"""Batched networks whose connections target part of the group (ranges that
start or end at odd neurons, a single neuron, ranges that do not meet a block's
first threads), with zero and longer delays, several events of a neuron in one
step and steps in which every neuron spikes: the same records and states as the
network alone, for block shapes with 4, 6 and 8 neurons per thread."""
import numpy as np
import pytest

import brian_b200 as b
from brian_b200 import ms, mV

pytestmark = pytest.mark.gpu


def _net(n, lo, hi, delayed, drive, mon):
    clk = b.Clock(dt=0.1 * ms)
    rng = np.random.default_rng(n + lo)
    P = b.NeuronGroup(n, model="dv/dt = (ge - v + %g*mV)/(10*ms) : volt\ndge/dt = -ge/(5*ms) : volt" % drive, threshold=10 * mV,
                      reset=0 * mV, clock=clk)
    P.v = rng.random(n) * 10 * mV
    T = P[lo:hi]
    objs = [P]
    for src, var, w in ((P, "ge", 0.3 * mV), (P[n // 3:], "v", -0.05 * mV)):
        m = len(src)
        row = np.arange(m + 1, dtype=np.int64) * min(6, hi - lo)
        cols = np.concatenate([np.sort(rng.choice(hi - lo, min(6, hi - lo), replace=False)) for _ in range(m)]).astype(np.int32)
        if delayed:
            C = b.DelayConnection(src, T, var, max_delay=1 * ms)
            C.connect_csr(row, cols, w, delay_steps=rng.integers(1, 11, len(cols)).astype(np.uint8))
        else:
            C = b.Connection(src, T, var)
            C.connect_csr(row, cols, w)
        objs.append(C)
    M = b.SpikeMonitor(P[mon:])
    return b.Network(*objs, M), P, M


CASES = [(700, 0, 700, False, 14, 0), (701, 1, 701, False, 14, 1), (701, 3, 4, True, 14, 33), (702, 255, 699, True, 14, 31),
         (511, 2, 509, False, 400, 0), (511, 7, 510, True, 400, 5)]


def _state(net, P, M):
    s, i = M._record()
    return [s.copy(), i.copy(), np.array(P.v), np.array(P.ge)] + [x.copy() for x in net._binding.rt.counters(1, 2)]


@pytest.mark.parametrize("shape,lanes", [(1, 32), (3, 8), (5, 16), (4, 4)])
def test_ranges(gpu_table, shape, lanes):
    b.clear()
    alone = [_net(*c) for c in CASES]
    for net, P, M in alone:
        net.run(20 * ms)
        net.run(5.3 * ms)
    want = [_state(*x) for x in alone]
    built = [_net(*c) for c in CASES]
    batch = b.NetworkBatch([x[0] for x in built])
    batch.set_shape(shape, lanes)
    batch.run(20 * ms)
    batch.run(5.3 * ms)
    assert sum(len(w[0]) for w in want) > 2000
    for c, w, x in zip(CASES, want, built):
        for p, q in zip(w, _state(*x)):
            assert np.array_equal(p, q), c
    batch.close()
    for x in built + alone:
        x[0]._invalidate()
