"""STDP on dense connections with pending postsynaptic updates: windows of
steps split by runs of odd lengths, weights, traces and spikes read and
weights written between runs, save and load in the middle of a window's
length, every update form and interaction, delays of either rule, subgroups,
FP32 and FP64 weights, sizes around the blocks -- bit for bit against the
oracle, which updates every step."""
import numpy as np
import pytest

import scenarios
import brian_b200 as b
from brian_b200 import Hz, ms, mV
from brian_b200.network import engine

pytestmark = pytest.mark.gpu


def _run(nin, nout, runs, wdtype=np.float32, update="additive", interactions="all", delay=0.0, sub=False,
         rates=(5.0, 60.0), drive=0.6, write=False, spread=False):
    b.clear()
    b.reinit_default_clock()
    rng = np.random.default_rng(nin + 3 * nout)
    eqs = b.Equations("dv/dt=(ge*(Ee-vr)+El-v)/taum : volt\ndge/dt=-ge/taue : 1", taum=10 * ms, taue=5 * ms,
                      Ee=0 * mV, vr=-60 * mV, El=-53 * mV)
    src = b.PoissonGroup(nin, rates=rng.uniform(*rates, nin) * Hz, seed=11)
    tgt = b.NeuronGroup(nout, model=eqs, threshold=-54 * mV, reset=-60 * mV)
    tgt.v = -60 * mV + 7 * mV * rng.random(nout)
    S, T = (src[nin // 5:nin - 3], tgt[nout // 4:nout - 1]) if sub else (src, tgt)
    gmax = drive / max(4, len(S)) * 30
    C = b.Connection(S, T, "ge", structure="dense", delay=delay, dtype=wdtype)
    W = rng.uniform(0, gmax, (len(S), len(T)))
    if spread:                                      # zeros, subnormal and tiny weights, and some past the bounds
        W[::3] *= 10.0 ** rng.integers(-46, 1, W[::3].shape)
        W[1::7] = 0.0
        W[2::11] = 3 * gmax
    C.connect(W=W)
    stdp = b.ExponentialSTDP(C, 20 * ms, 15 * ms, 0.02, -0.021, wmax=gmax, interactions=interactions, update=update)
    M = b.SpikeMonitor(tgt)
    net = b.Network(src, tgt, C, stdp, M)
    out = {}
    for k, n in enumerate(runs):
        net.run(n * 0.1 * ms)
        out["W%d" % k] = C._weights().astype(np.float64).copy()
        a, p = stdp._traces()
        out["pre%d" % k], out["post%d" % k] = a.copy(), p.copy()
        if write and k == 0:
            C._set_weights(np.minimum(C._weights() * 1.25 + gmax / 64, gmax))
    out.update(scenarios._result(net, groups=[tgt], spikemons=[M]))
    net._invalidate()
    return out


def _both(oracle_table, **kw):
    with engine(oracle_table):
        ref = _run(**kw)
    gpu = _run(**kw)
    assert len(ref["spk0.idx"]) > 0 or sum(kw["runs"]) < 40
    for k in ref:
        assert np.array_equal(ref[k], gpu[k]), k


@pytest.mark.parametrize("runs", [(1, 1, 2), (31, 32, 33), (63, 64, 65), (97, 200, 5), (1056,)])
def test_windows(oracle_table, gpu_table, runs):
    _both(oracle_table, nin=300, nout=70, runs=runs)


@pytest.mark.parametrize("nin,nout", [(1, 1), (31, 33), (32, 32), (33, 31), (8, 257), (1025, 5), (40, 300)])
def test_sizes(oracle_table, gpu_table, nin, nout):
    _both(oracle_table, nin=nin, nout=nout, runs=(150, 90), rates=(200.0, 900.0), drive=2.0)


@pytest.mark.parametrize("update", ["additive", "multiplicative", "mixed"])
@pytest.mark.parametrize("interactions", ["all", "nearest", "nearest_pre", "nearest_post"])
def test_forms(oracle_table, gpu_table, update, interactions):
    _both(oracle_table, nin=200, nout=40, runs=(130, 70), wdtype=np.float64, update=update, interactions=interactions)


@pytest.mark.parametrize("wdtype", [np.float32, np.float64])
def test_subgroups_and_written_weights(oracle_table, gpu_table, wdtype):
    _both(oracle_table, nin=250, nout=66, runs=(75, 110), wdtype=wdtype, sub=True, write=True)


def test_homogeneous_delay(oracle_table, gpu_table):
    _both(oracle_table, nin=200, nout=40, runs=(75, 110), delay=0.7 * ms)


def test_small_and_outlying_weights(oracle_table, gpu_table):
    """Weights from 0 and the subnormals to above wmax."""
    _both(oracle_table, nin=240, nout=48, runs=(90, 70), spread=True, drive=1.0)


def test_many_spikes_a_step(oracle_table, gpu_table):
    """More spiking rows than one list of a block holds, and than one pass of its history words."""
    _both(oracle_table, nin=40000, nout=3, runs=(40,), rates=(900.0, 1100.0), drive=1.0)
