"""Which kernel runs a small network -- one block, a thread-block cluster, the
persistent kernel or stepped launches -- and that each gives the oracle's run;
a device that places no cluster among them."""
import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu


def _run(n, k, refuse=False, **model):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(n)
    P = b.NeuronGroup(n, model="dv/dt = (ge + 12*mV - v)/(20*ms) : volt\ndge/dt = -ge/(5*ms) : volt", threshold=10 * mV,
                      reset=0 * mV, **model)
    offs = rng.choice(n, k, replace=False)              # k synapses from and to every neuron
    cols = np.sort((np.arange(n)[:, None] + offs) % n, axis=1).astype(np.int32).ravel()
    C = b.Connection(P, P, "ge")
    C.connect_csr(np.arange(n + 1, dtype=np.int64) * k, cols, 4 * mV / k)
    P.v = rng.random(n) * 10 * mV
    M = b.SpikeMonitor(P)
    net = b.Network(P, C, M)
    net.prepare(configure=(lambda rt: rt.debug_refuse_cluster()) if refuse else None)
    net.run(10 * ms)
    out = scenarios._result(net, groups=[P], spikemons=[M])
    st = net.stats()
    net._invalidate()
    return out, (st.get("cluster_blocks"), st.get("cluster_npt"), st.get("persistent_threads"))


# neurons, synapses a neuron, blocks and neurons per thread of the cluster kernel (0: another kernel).  More than 2^18 - 1
# synapses into one block do not fit its transaction count; one block has none and no such limit.
SHAPES = [(512, 20, 1, 1), (2048, 20, 1, 4), (2049, 20, 5, 1), (8193, 20, 9, 2), (2000, 600, 1, 4), (3000, 511, 6, 1), (3000, 512, 0, 0),
          (33000, 9, 0, 0)]


@pytest.mark.parametrize("n,k,blocks,npt", SHAPES)
@pytest.mark.parametrize("model", [{}, dict(method="Euler")])
def test_kernel(oracle_table, gpu_table, n, k, blocks, npt, model):
    with engine(oracle_table):
        ref, _ = _run(n, k, **model)
    for refuse in (False, True):
        gpu, ran = _run(n, k, refuse, **model)
        if refuse or not blocks:
            assert ran == (0, 0, 0 if model else 512)
        else:
            assert ran == (blocks, npt, 512)
        scenarios.compare(ref, gpu)
    assert len(ref["spk0.idx"]) > n // 20


def test_forced_persistent_kernel(gpu_table):
    b.set_global_preferences(persistent=512)
    try:
        assert _run(3000, 20)[1] == (0, 0, 512)
    finally:
        b.set_global_preferences(persistent=True)
