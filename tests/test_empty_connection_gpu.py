"""A group with a Connection onto itself that has no synapses (and one that
has some): every route runs it like the oracle."""
import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu


def _net(n, full, **model):
    P = b.NeuronGroup(n, model="dv/dt = (20*mV-v)/(10*ms) : volt", threshold=10 * mV, reset=0 * mV,
                      clock=b.Clock(dt=0.1 * ms), **model)
    P.v = np.linspace(0, 9.9, n) * mV
    C = [b.Connection(P, P, "v")]
    if full:
        C.append(b.Connection(P, P, "v"))
        C[1].connect_csr(np.arange(n + 1, dtype=np.int64), np.roll(np.arange(n, dtype=np.int32), 1), 0.1 * mV)
    M = b.SpikeMonitor(P)
    return b.Network(P, *(C + [M])), P, C, M


def _run(n, full, batch=False, **model):
    b.clear()
    b.reinit_default_clock()
    net, P, C, M = _net(n, full, **model)
    (b.NetworkBatch([net]) if batch else net).run(30 * ms)
    assert len(C[0]._weights()) == 0
    out = scenarios._result(net, groups=[P], spikemons=[M])
    net._invalidate()
    return out


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n,persistent", [(300, True), (3000, True), (3000, 512), (3000, False)])
@pytest.mark.parametrize("model", [{}, dict(method="Euler")])
def test_routes(oracle_table, gpu_table, n, persistent, full, model):
    with engine(oracle_table):
        ref = _run(n, full, **model)
    b.set_global_preferences(persistent=persistent)
    try:
        gpu = _run(n, full, **model)
    finally:
        b.set_global_preferences(persistent=True)
    assert len(ref["spk0.idx"]) > n
    scenarios.compare(ref, gpu)


@pytest.mark.parametrize("full", [False, True])
def test_batch(oracle_table, gpu_table, full):
    with engine(oracle_table):
        ref = _run(700, full)
    scenarios.compare(ref, _run(700, full, batch=True))
