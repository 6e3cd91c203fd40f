"""The proposer network's tiles at their edges, against the CPU oracle.

Rows: one, around the 32-row tile, odd, and enough for the 64-row tile (from 296
of its tiles on).  Bounds as for the ordinary size: the device rounds to BF16 where
the oracle (bf16_ops) does, so outputs agree to 1e-3 of the largest, and the
gradient of each layer to 2e-2 of its norm (a value next to a rounding boundary
moves by 2^-8).  The first Adam step is lr g / (|g| + eps): its FP32 rounding is a
few 1e-7 of the step and 6e-8 of the parameter.
"""
import numpy as np
import pytest

from kalnajs_log_spirals_b200 import proposer as P
from oracle import np_mlp as O

pytestmark = pytest.mark.gpu


def check(mlp, X, T, width, depth):
    params = mlp.params()
    Y = mlp.forward(X)
    g, loss = mlp.grad(X, T)
    Ye, le, ge = O.forward_backward(params, X, T, width, depth, bf16_ops=True)
    assert Y.shape == Ye.shape
    assert np.max(np.abs(Y - Ye)) <= 1e-3 * np.max(np.abs(Ye))
    assert abs(loss - le) <= 1e-3 * le
    o = 0
    for di, do in O.layer_shapes(width, depth):
        for n in (di * do, do):
            assert np.linalg.norm(g[o:o + n] - ge[o:o + n]) <= 2e-2 * np.linalg.norm(ge[o:o + n])
            o += n
    return params, g, loss


@pytest.mark.parametrize("width,depth,n", [
    (256, 4, 1), (256, 4, 31), (16, 2, 33), (48, 3, 77), (256, 4, 1024), (112, 5, 1001),
    (256, 3, 4800), (48, 3, 19001)])
def test_mlp_sizes(lib_path, width, depth, n):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 5)).astype(np.float32)
    T = rng.normal(size=(n, 3)).astype(np.float32)
    mlp = P.MLP(width, depth, seed=n + 1)
    p, g, loss = check(mlp, X, T, width, depth)
    # one step over all rows (in shuffled order), then the new BF16 copies
    lr = 1e-3
    hist = mlp.train(X, T, epochs=1, batch=n, lr=lr, seed=2)
    assert abs(hist[0] - loss) <= 1e-5 * loss
    q = mlp.params()
    big = np.abs(g) > 1e-3 * np.abs(g).max()
    step = lr * g / (np.abs(g) + 1e-8)
    assert np.all(np.abs(q - (p - step))[big] <= 1e-5 * lr + 2e-7 * np.abs(p[big]))
    check(mlp, X, T, width, depth)
    mlp.close()


def test_mlp_steps_of_an_epoch(lib_path):
    """An epoch's steps follow one another: the first batch of a one-step epoch and
    of a longer one is the same, and a remainder below the batch is left out."""
    rng = np.random.default_rng(5)
    X = rng.normal(size=(199, 5)).astype(np.float32)
    T = rng.normal(size=(199, 3)).astype(np.float32)
    a, b = P.MLP(64, 3, seed=1), P.MLP(64, 3, seed=1)
    ha = a.train(X, T, epochs=2, batch=50, lr=1e-3, seed=3)
    hb = [b.train(X, T, epochs=1, batch=50, lr=1e-3, seed=3)[0]]
    assert ha[0] == hb[0] and len(ha) == 2 and np.isfinite(ha).all()
    check(a, X, T, 64, 3)
    a.close()
    b.close()


def test_mlp_training_set_in_segments(lib_path):
    """More rows than are kept on the device (2^22): segments in the epoch's order.
    With lr = 0 the epoch's loss is that of all rows but the one left out (FP32 sums of
    4e6 terms: 1e-4), and one step over all of the rows is the gradient's."""
    n = (1 << 22) + 1
    rng = np.random.default_rng(9)
    X = rng.normal(size=(n, 5)).astype(np.float32)
    T = rng.normal(size=(n, 3)).astype(np.float32)
    mlp = P.MLP(16, 2, seed=4)
    p = mlp.params()
    g, loss = mlp.grad(X, T)
    hist = mlp.train(X, T, epochs=2, batch=1 << 20, lr=0.0, seed=1)
    assert np.array_equal(mlp.params(), p)
    assert np.all(np.abs(hist - loss) <= 1e-4 * loss)
    mlp.close()
    mlp = P.MLP(16, 2, seed=4)                 # (Adam's moments at zero)
    mlp.train(X, T, epochs=1, batch=n, lr=1e-3, seed=1)
    q = mlp.params()
    big = np.abs(g) > 1e-2 * np.abs(g).max()
    step = 1e-3 * g / (np.abs(g) + 1e-8)
    assert np.all(np.abs(q - (p - step))[big] <= 1e-8 + 2e-7 * np.abs(p[big]))
    mlp.close()
