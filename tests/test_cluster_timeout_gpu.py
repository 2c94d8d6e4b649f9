"""The cluster kernel's bounded waits: one block holds back its arrivals, every
wait runs out, the run ends with BG_ETIMEOUT within its limit (all pushes of the
blocks to one another landed), the network refuses to go on and the device runs
the next one like the oracle."""
import time

import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200._lib import EngineError
from brian_b200.network import engine

pytestmark = pytest.mark.gpu

BG_ETIMEOUT, BG_ESTATE = -4, -6


def _net(n, kind, model):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(n)
    P = b.NeuronGroup(n, model="dv/dt = (ge + 12*mV - v)/(20*ms) : volt\ndge/dt = -ge/(5*ms) : volt", threshold=10 * mV,
                      reset=0 * mV, **model)
    cols = np.concatenate([np.sort(rng.choice(n, 40, replace=False)) for _ in range(n)]).astype(np.int32)
    ptr = np.arange(n + 1, dtype=np.int64) * 40
    if kind == "delay":
        C = b.DelayConnection(P, P, "ge", max_delay=1 * ms)
        C.connect_csr(ptr, cols, 0.1 * mV, delay_steps=rng.integers(1, 11, len(cols)).astype(np.uint8))
    else:
        C = b.Connection(P, P, "ge")
        C.connect_csr(ptr, cols, 0.1 * mV)
    P.v = 8 * mV + rng.random(n) * 4 * mV            # half of the neurons spike in the first steps
    M = b.SpikeMonitor(P)
    return b.Network(P, C, M), P, M


@pytest.mark.parametrize("n,block", [(3000, 0), (3000, 5), (9000, 3), (30000, 14)])
@pytest.mark.parametrize("kind", ["connection", "delay"])
@pytest.mark.parametrize("steps", [1, 2, 100])
@pytest.mark.parametrize("model", [{}, dict(method="Euler")])
def test_wait_runs_out(oracle_table, gpu_table, n, block, kind, steps, model):
    b.set_global_preferences(spin_limit=20000)       # at most 20 ms a wait
    try:
        net, P, M = _net(n, kind, model)
        net.prepare(configure=lambda rt: rt.debug_hold_cluster(block))
        assert net.stats()["cluster_blocks"] > block
        t0 = time.perf_counter()
        with pytest.raises(EngineError) as e:
            net.run(steps * 0.1 * ms)
        assert e.value.code == BG_ETIMEOUT, e.value
        assert time.perf_counter() - t0 < 2.0        # a wait in the loop or after it, one for the pushes of each mbarrier
        with pytest.raises(EngineError) as e:
            net.run(0.1 * ms)
        assert e.value.code == BG_ESTATE
        net._invalidate()
    finally:
        b.set_global_preferences(spin_limit=None)
    outs = []
    for table in (oracle_table, None):
        if table is None:
            net, P, M = _net(n, kind, model)
            net.run(2 * ms)
            assert net.stats()["cluster_blocks"] > block
        else:
            with engine(table):
                net, P, M = _net(n, kind, model)
                net.run(2 * ms)
        outs.append(scenarios._result(net, groups=[P], spikemons=[M]))
        net._invalidate()
    scenarios.compare(*outs)
