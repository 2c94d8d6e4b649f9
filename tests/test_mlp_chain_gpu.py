"""The proposal network's fused layer chains and the one-launch weight
gradients at the sizes where they can go wrong: one row tile, a last tile of
one row, more row tiles than SMs (a block takes a second tile into the buffer
the first one's stores read), the smallest batch of a training step (one K
chunk per split) and outputs that fill a part, one or several of the loss
kernel's groups."""
import numpy as np
import pytest

from brian_b200 import _lib
from oracle import mlp as om

pytestmark = pytest.mark.gpu


def _net(ydim, seed):
    rng = np.random.default_rng(seed)
    P = om.init_params(rng)
    for l in range(4):
        P[l] = (P[l][0], (0.1 * rng.standard_normal(om.ROWS[l])).astype(np.float32))
    P[3][0][2 * ydim:] = 0
    P[3][1][2 * ydim:] = 0
    h = _lib.MLPHandle(ydim)
    for l in range(4):
        h.set_params(l, *P[l])
    return h, P, rng


@pytest.mark.parametrize("n", [1, 128, 129, 128 * 148 + 1, 128 * 300])
def test_forward_rows_do_not_depend_on_the_batch(n):
    # every row's products are summed in one order whatever tile, block or
    # pass it falls in, so a batch equals its pieces bit for bit
    h, P, rng = _net(5, 3)
    X = rng.standard_normal((n, 64)).astype(np.float32)
    out = h.forward(X)
    step = 128 * 37
    for r in range(0, n, step):
        assert np.array_equal(out[r:r + step], h.forward(X[r:r + step])), r
    _, ref = om.forward(P, X[-300:])
    # bf16 operands (8 bits) through four layers against the oracle's own order
    assert np.max(np.abs(out[-300:] - ref[:, :10])) < 2e-2 * max(1.0, np.max(np.abs(ref)))
    h.close()


@pytest.mark.parametrize("n,ydim", [(512, 5), (512, 1), (1024, 32), (1536, 7), (128 * 152, 5)])
def test_gradients(n, ydim):
    h, P, rng = _net(ydim, n + ydim)
    X = rng.standard_normal((n, 64)).astype(np.float32)
    Y = rng.uniform(-1, 1, (n, ydim)).astype(np.float32)
    h.set_data(X, Y)
    loss, dW, db = h.gradients(n)
    rloss, rdW, rdb, _ = om.gradients(P, X, Y, ydim)
    assert abs(loss - rloss) <= 1e-3 * abs(rloss)
    for l in range(4):
        # both sides round activations and gradients to bf16; sums of another
        # order flip some of those roundings (2^-9 of an entry each)
        assert np.linalg.norm(dW[l] - rdW[l]) < 2e-2 * np.linalg.norm(rdW[l]), l
        assert np.linalg.norm(db[l] - rdb[l]) < 2e-2 * np.linalg.norm(rdb[l]), l
    assert np.all(dW[3][2 * ydim:] == 0) and np.all(db[3][2 * ydim:] == 0)
    # again on the same buffers, and after another batch size in between
    again = h.gradients(n)
    h.forward(X[:200])
    third = h.gradients(n)
    for l in range(4):
        assert np.array_equal(dW[l], again[1][l]) and np.array_equal(dW[l], third[1][l])
        assert np.array_equal(db[l], again[2][l]) and np.array_equal(db[l], third[2][l])
    h.close()
