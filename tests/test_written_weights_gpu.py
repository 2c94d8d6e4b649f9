"""Weights of a prepared network's zero-delay Connections written between runs
-- another shared value, unequal values, equal ones again -- on every route the
network may take (the cluster kernel with one and several blocks, the
persistent kernel, stepped launches; linear and generated models): bit for bit
the oracle's run.  A batch refuses a network whose weights are no longer shared."""
import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200._lib import EngineError
from brian_b200.network import engine

pytestmark = pytest.mark.gpu

BG_ENOSYS = -7
CONST = dict(taum=20 * ms, taue=5 * ms, El=-49 * mV)


def _net(n, mixed=False, seed=4, **model):
    rng = np.random.default_rng(seed + n)
    P = b.NeuronGroup(n, model=b.Equations("dv/dt = (ge-(v-El))/taum : volt\ndge/dt = -ge/taue : volt", **CONST),
                      threshold=-50 * mV, reset=-60 * mV, clock=b.Clock(dt=0.1 * ms), **model)
    conns = []
    for k, (src, w) in enumerate(((P, 0.4 * mV), (P.subgroup(n // 4), -0.7 * mV))):
        cols = np.concatenate([np.sort(rng.choice(n, 9, replace=False)) for _ in range(len(src))]).astype(np.int32)
        ptr = np.arange(len(src) + 1, dtype=np.int64) * 9
        if mixed and k == 1:
            C = b.DelayConnection(src, P, "ge", max_delay=1 * ms)
            C.connect_csr(ptr, cols, w, delay_steps=rng.integers(1, 11, len(cols)).astype(np.uint8))
        else:
            C = b.Connection(src, P, "ge")
            C.connect_csr(ptr, cols, w)
        conns.append(C)
    P.v = -60 * mV + rng.random(n) * 14 * mV
    M = b.SpikeMonitor(P)
    return b.Network(P, *(conns + [M])), P, conns, M


def _run(n, mixed=False, **model):
    b.clear()
    b.reinit_default_clock()
    net, P, conns, M = _net(n, mixed, **model)
    C, W = conns[0], conns[0]._nnz()
    rng = np.random.default_rng(9)
    net.run(5 * ms)
    for w in (np.full(W, 0.9 * mV), rng.uniform(-0.2, 1.2, W) * mV, rng.uniform(-0.2, 1.2, W) * mV, np.full(W, 0.5 * mV)):
        C._set_weights(w)
        assert np.array_equal(C._weights(), w)
        net.run(5 * ms)
    row, col = 2, int(C._cols[C._rowptr[2]])
    C[row, col] = 2 * mV                    # one element
    net.run(5 * ms)
    out = scenarios._result(net, groups=[P], spikemons=[M])
    net._invalidate()
    return out


@pytest.mark.parametrize("n,persistent,mixed", [(400, True, False), (3000, True, False), (3000, True, True), (3000, 512, False),
                                                (40000, True, False), (3000, False, False)])
@pytest.mark.parametrize("model", [{}, dict(method="Euler")])
def test_routes(oracle_table, gpu_table, n, persistent, mixed, model):
    with engine(oracle_table):
        ref = _run(n, mixed, **model)
    b.set_global_preferences(persistent=persistent)
    try:
        gpu = _run(n, mixed, **model)
    finally:
        b.set_global_preferences(persistent=True)
    assert len(ref["spk0.idx"]) > 50
    scenarios.compare(ref, gpu)


def test_batch(gpu_table):
    """A batch takes another shared value and refuses unequal ones."""
    outs = []
    for batched in (True, False):
        b.clear()
        parts = [_net(500, seed=k) for k in range(3)]
        nets = [p[0] for p in parts]
        batch = b.NetworkBatch(nets)
        run = batch.run if batched else lambda t: [net.run(t) for net in nets]
        run(5 * ms)
        C = parts[1][2][0]
        C._set_weights(np.full(C._nnz(), 0.8 * mV))
        run(5 * ms)
        outs.append([np.array(getattr(p[1], v)) for p in parts for v in ("v", "ge")])
        if batched:
            W = C._weights()
            W[5] *= 2
            C._set_weights(W)
            with pytest.raises(EngineError) as e:
                batch.run(5 * ms)
            assert e.value.code == BG_ENOSYS, e.value
        for net in nets:
            net._invalidate()
    assert all(np.array_equal(x, y) for x, y in zip(*outs))
