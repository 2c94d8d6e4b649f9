"""The fitting kernel's division forms and its task queue, bit for bit.

Candidates of one warp whose dividends are ordinary, infinite, NaN, zero (with
divisors of either sign) or subnormal take the fast form, the wide form and
IEEE division by turns; every state must equal numpy's arithmetic in the
scalar type exactly (each form is RN(a/b), so the tolerance is zero).  More
tasks than the queue has single classes must each run exactly once."""
import numpy as np
import pytest

import test_fit_gpu as tf
from brian_b200 import Equations
from brian_b200.codegen import generate_model_code
from oracle import fitting as of

pytestmark = pytest.mark.gpu
DT = tf.DT


def _case(S0, I, nsteps):
    ns = S0.shape[1]
    last = int(np.max(nsteps))
    return dict(S0=S0, I=I, I_offset=np.zeros(ns, int), nsteps=np.broadcast_to(nsteps, (ns,)).copy(),
                spiketimes=np.array([-10000, last + 10000]), spk_offset=np.zeros(ns, int),
                spk_end=np.full(ns, 2), delay=np.zeros(ns, int), refractory=np.zeros(ns, int))


def _check(eqs, thr, rst, c, precision):
    dtype = np.float32 if precision == 32 else np.float64
    code = generate_model_code(eqs, thr, rst, DT, scalar="float" if precision == 32 else "double")
    h = tf._device(code, c, precision, True)
    h.run(0, int(c["nsteps"].max()))
    coinc, nspk, S = h.read(state=True)
    m = of.ModelOracle(eqs, thr, rst, DT, dtype)
    with np.errstate(all="ignore"):
        r = of.simulate(m, c["S0"], c["I"], c["I_offset"], c["nsteps"], c["spiketimes"], c["spk_offset"],
                        c["spk_end"], refractory=c["refractory"])
    assert np.array_equal(S, r["state"], equal_nan=True)
    assert np.array_equal(np.signbit(S), np.signbit(r["state"])) or np.isnan(S).any()
    assert np.array_equal(nspk, r["nspikes"])
    return S


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("refr", [0, 7])
@pytest.mark.parametrize("steps", [31, 32, 45, 3000])
def test_odd_dividends(precision, refr, steps):
    rng = np.random.default_rng(steps + precision + refr)
    ns = 67                                           # two whole warps and three lanes
    tau = rng.uniform(2e-3, 2e-2, ns)
    tau[3::8] *= -1                                   # runs off to infinity (or spikes) and stays there
    tau[5::16] = -2e-4                                # ... within a few steps
    V0 = rng.uniform(-1, 1, ns)
    a = rng.uniform(-1, 2, ns)
    V0[::11] = a[::11]                                # zero dividends, divisors of either sign
    V0[7] = np.inf
    V0[40] = np.nan
    V0[20] = 1e-36 if precision == 32 else 1e-300     # decays through the subnormals
    a[20] = 0.0
    V0[21] = -3e38 if precision == 32 else -1.5e308   # close to overflow
    tau[21] = 1e-3
    S0 = np.vstack([V0, a, tau])
    c = _case(S0, rng.uniform(-0.1, 0.1, steps), np.full(ns, steps))
    c["refractory"] = np.full(ns, refr)
    eqs = Equations("dV/dt = (a + I - V)/tau : 1\nI : 1\na : 1\ntau : 1", dummy=0.0)
    S = _check(eqs, "V > 1.0", "V = 0", c, precision)
    if steps == 3000:
        assert np.isinf(S[0]).any()                   # some candidate did reach infinity


def test_more_tasks_than_classes():
    rng = np.random.default_rng(4)
    ns = 32 * 148 * 70 + 5                            # 64 classes of one task per SM, and more
    S0 = np.vstack([rng.uniform(-1, 0, ns), rng.uniform(0, 1, ns), rng.uniform(1e-3, 1e-2, ns)])
    c = _case(S0, rng.uniform(0, 0.1, 3), rng.integers(0, 4, ns))
    eqs = Equations("dV/dt = (a + I - V)/tau : 1\nI : 1\na : 1\ntau : 1", dummy=0.0)
    _check(eqs, "V > 0.5", "V = 0", c, 32)
