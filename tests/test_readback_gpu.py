"""Results read back from the device: spike records of the persistent kernels
with none, few, more than one pinned block of and more than the monitor's
buffer of records, and weights of sizes around the pinned blocks, in the
connection's own type and widened, before and after prepare and from two
threads at once."""
import threading

import numpy as np
import pytest

import brian_b200 as b
from brian_b200 import ms, mV

pytestmark = pytest.mark.gpu


def _firing(n, fire):
    """n neurons that fire in every step if `fire`, never otherwise."""
    b.clear()
    b.reinit_default_clock()
    P = b.NeuronGroup(n, model=b.Equations("dv/dt = -(v+49*mV)/(20*ms) : volt"), threshold=-70 * mV if fire else 0 * mV,
                      reset=-60 * mV)
    P.v = -60 * mV
    C = b.Connection(P, P, "v")
    C.connect_csr(np.arange(n + 1, dtype=np.int64), ((np.arange(n) + 1) % n).astype(np.int32), 0.0)
    M = b.SpikeMonitor(P)
    return b.Network(P, C, M), M


@pytest.mark.parametrize("n,steps,fire", [(500, 70, False), (3, 1, True), (64, 1024, True), (4000, 100, True), (512, 1500, True),
                                          (40000, 1000, True)])
def test_spike_records(n, steps, fire):
    # (64 x 1024 records fill a block's share exactly, 4000 x 100 pass it,
    # 512 x 1500 are two launches, 40000 x 1000 pass the monitor's buffer)
    net, M = _firing(n, fire)
    net.run(steps * 0.1 * ms)
    assert net._binding.rt.stats()["persistent_threads"] > 0
    s, i = M._record()
    if not fire:
        assert len(s) == 0 and len(i) == 0
        return
    assert len(s) == n * steps
    assert np.array_equal(i.reshape(steps, n), np.broadcast_to(np.arange(n, dtype=np.int32), (steps, n)))
    assert np.array_equal(s.reshape(steps, n)[:, 0], np.arange(steps)) and np.array_equal(s.reshape(steps, n)[:, -1], np.arange(steps))
    # a second run's records follow
    if n * steps < 1000000:
        net.run(2 * 0.1 * ms)
        s, i = M._record()
        assert len(s) == n * (steps + 2) and s[-1] == steps + 1 and i[-1] == n - 1


def _dense(ns, nt, dtype, seed):
    A = b.NeuronGroup(ns, model=b.Equations("dv/dt = -v/(20*ms) : volt"))
    B = b.NeuronGroup(nt, model=b.Equations("dv/dt = -v/(20*ms) : volt"))
    C = b.Connection(A, B, "v", structure="dense")
    W = np.random.default_rng(seed).random((ns, nt)).astype(dtype)
    C.connect(A, B, W)
    return b.Network(A, B, C), C, W


@pytest.mark.parametrize("ns,nt", [(1, 1), (37, 53), (1024, 128), (1237, 1999), (2048, 1024)])
def test_weights(ns, nt):
    b.clear()
    b.reinit_default_clock()
    net, C, W = _dense(ns, nt, np.float64, ns)
    net.run(0.2 * ms)
    rt, cid = net._binding.rt, net._binding.cids[C]
    got = rt.conn_read_weights(cid, ns * nt, C.dtype)
    assert got.dtype == C.dtype and np.array_equal(got.reshape(ns, nt), W.astype(C.dtype))
    assert np.array_equal(rt.conn_get_weights(cid, ns * nt), got.astype(np.float64))
    with pytest.raises(Exception):
        rt.conn_read_weights(cid, ns * nt + 1, C.dtype)


def test_weights_from_two_threads():
    b.clear()
    b.reinit_default_clock()
    made = [_dense(1800, 1500, np.float64, k) for k in range(2)]
    for net, _, _ in made:
        net.run(0.2 * ms)
    bad = []

    def read(k):
        net, C, W = made[k]
        for _ in range(5):
            if not np.array_equal(np.asarray(C._weights()).reshape(W.shape), W.astype(C.dtype)):
                bad.append(k)

    th = [threading.Thread(target=read, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
