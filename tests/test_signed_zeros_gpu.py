"""States of -0.0 on the persistent routes: the update's sums start from +0 and
a DelayConnection adds its row also where no event is due, so the sign of a
zero is the oracle's (and the stepped launches') too."""
import numpy as np
import pytest

import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu


def _run(n, kind, method, steps):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(n)
    # v spikes now and then; x and y are multiples of themselves
    P = b.NeuronGroup(n, model="dv/dt = (12*mV + x + y - v)/(10*ms) : volt\ndx/dt = -x/(5*ms) : volt\ndy/dt = 0*y/ms : volt"
                      if method else "dv/dt = (x - y - v)/(10*ms) : volt\ndx/dt = -x/(5*ms) : volt\ndy/dt = -y/(7*ms) : volt",
                      threshold=10 * mV, reset=-0.0 * mV, **(dict(method=method) if method else {}))
    T = P[n // 3:n - n // 5]
    objs = [P]
    for var in ("x", "y"):
        cols = np.concatenate([np.sort(rng.choice(len(T), 2, replace=False)) for _ in range(n)]).astype(np.int32)
        ptr = np.arange(n + 1, dtype=np.int64) * 2
        if kind == "delay":
            C = b.DelayConnection(P, T, var, max_delay=1 * ms)
            C.connect_csr(ptr, cols, 0.01 * mV, delay_steps=rng.integers(1, 11, len(cols)).astype(np.uint8))
        else:
            C = b.Connection(P, T, var)
            C.connect_csr(ptr, cols, 0.01 * mV)
        objs.append(C)
    P.v = np.where(np.arange(n) % 97 == 0, 11 * mV, -0.0)
    P.x = np.where(rng.random(n) < 0.5, -0.0, 0.0)
    P.y = np.where(rng.random(n) < 0.5, -0.0, 0.0)
    net = b.Network(*objs)
    net.run(steps * 0.1 * ms)
    out = [np.array(getattr(P, v)) for v in "vxy"]
    net._invalidate()
    return out


@pytest.mark.parametrize("method", [None, "Euler"])
@pytest.mark.parametrize("kind", ["connection", "delay"])
@pytest.mark.parametrize("n,persistent", [(500, True), (3000, True), (3000, 512), (3000, False)])
@pytest.mark.parametrize("steps", [1, 15])
def test_signs(oracle_table, gpu_table, n, persistent, kind, method, steps):
    with engine(oracle_table):
        ref = _run(n, kind, method, steps)
    b.set_global_preferences(persistent=persistent)
    try:
        gpu = _run(n, kind, method, steps)
    finally:
        b.set_global_preferences(persistent=True)
    for r, g in zip(ref, gpu):
        assert np.array_equal(r, g) and np.array_equal(np.signbit(r), np.signbit(g))
