"""Pending postsynaptic updates of a dense connection (ExponentialSTDP, FP32
weights) where a weight or a trace is a special value, against the oracle,
which updates every step: equal down to the sign of a zero and NaN for NaN."""
import numpy as np
import pytest

import brian_b200 as b
from brian_b200 import ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu

NIN, NOUT = 41, 70          # a band of one row at the end; columns past two warps


def _run(W, Ap, Am, wmax, gap, wmin=0.0):
    """Some sources spike before, some between and some after the targets'
    spikes; a weight's pending updates are applied by the pass at the end of a
    run where its source stays silent, else when it spikes."""
    b.clear()
    b.reinit_default_clock()
    step = 0.1 * ms
    rng = np.random.default_rng(3)
    # sources 0-9 never spike, 10-19 in the first run only, 20-29 also late in the
    # gap (their weights meet the targets' trace as it is by then), the others in the last run
    spikes = [(int(i), (2 + int(k)) * step) for i in range(10, NIN) for k in rng.integers(0, 25, 3)]
    last = 40 + gap
    spikes += [(int(i), (last - 5 - int(k)) * step) for i in range(20, 30) for k in rng.integers(0, 20, 2)]
    spikes += [(int(i), (last + 5 + int(k)) * step) for i in range(30, NIN) for k in rng.integers(0, 20, 2)]
    src = b.SpikeGeneratorGroup(NIN, spikes)
    tgt = b.NeuronGroup(NOUT, model="dv/dt = -v/(10*ms) : volt\ndge/dt = -ge/(5*ms) : 1", threshold=1 * mV, reset=0 * mV)
    C = b.Connection(src, tgt, "ge", structure="dense", dtype=np.float32)
    C.connect(W=W)
    with np.errstate(all="ignore"):
        stdp = b.STDP(C, eqs="dA_pre/dt = -A_pre/(1*ms) : 1\ndA_post/dt = -A_post/(1*ms) : 1", pre="A_pre += Ap\nw += A_post",
                      post="A_post += Am\nw += A_pre", wmin=wmin, wmax=wmax)
    net = b.Network(src, tgt, C, stdp)
    out = []
    for n in (40, gap, 60):
        for part in (1, n - 1):
            # every other target spikes at the start of each run, all of them in its second step
            tgt.v = np.where((np.arange(NOUT) % 2 == 0) | (part > 1), 2 * mV, 0.0) if n != gap else 0 * mV
            net.run(part * step)
        out += [C._weights().copy(), stdp._traces()[0].copy(), stdp._traces()[1].copy()]
    net._invalidate()
    return out


def _w(kind):
    rng = np.random.default_rng(7)
    W = rng.uniform(0.0, 0.01, (NIN, NOUT)).astype(np.float32)
    z = rng.random(W.shape)
    if kind == "negative zeros":
        W[z < 0.4] = -0.0
    elif kind == "zeros":
        W[:] = 0.0
    elif kind == "infinite":
        W[z < 0.2], W[z > 0.8] = np.inf, -np.inf
    elif kind == "nan":
        W[z < 0.3] = np.nan
    elif kind == "large":
        W[z < 0.3] = 3.4e38
    elif kind == "tiny":
        W = (W * 10.0 ** rng.integers(-44, -20, W.shape)).astype(np.float32)
    return W


# weights, Ap, Am, wmax, steps between the targets' spikes (1200: a trace of 1 ms falls below 2^-150)
CASES = [("negative zeros", 1e-4, -1.05e-4, 0.01, 40), ("zeros", 1e-4, -1.05e-4, 0.01, 1200), ("zeros", -1e-4, 1e-4, 0.01, 1200),
         ("plain", -1e-4, 1e-4, 0.01, 1200), ("tiny", -1e-40, 1e-40, 0.01, 40), ("plain", np.nan, -1e-4, 0.01, 40),
         ("plain", np.inf, -1e-4, 0.01, 40), ("plain", -np.inf, 1e-4, 0.01, 40), ("nan", 1e-4, -1e-4, 0.01, 40),
         ("infinite", -2e38, 1e-4, np.inf, 40), ("large", 3e37, -1e-4, np.inf, 40), ("large", -3e37, 2e37, np.inf, 40)]


@pytest.mark.parametrize("kind,Ap,Am,wmax,gap", CASES)
@pytest.mark.parametrize("wmin", [0.0, -0.0, -1e-3])
def test_special_values(oracle_table, gpu_table, kind, Ap, Am, wmax, gap, wmin):
    with engine(oracle_table):
        ref = _run(_w(kind), Ap, Am, wmax, gap, wmin)
    gpu = _run(_w(kind), Ap, Am, wmax, gap, wmin)
    for r, g in zip(ref, gpu):
        assert np.array_equal(r, g, equal_nan=True)
        assert np.array_equal(np.signbit(r)[~np.isnan(r)], np.signbit(g)[~np.isnan(g)])
