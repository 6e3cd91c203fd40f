"""Gradients of a batch whose training buffers do not all fit beside one another: the
buffers of one layer at a time, with the same bits."""
import numpy as np
import pytest
import torch

from kalnajs_log_spirals_b200 import proposer as P

pytestmark = pytest.mark.gpu


def test_gradients_with_little_memory(lib_path):
    """Width 256, depth 16: 14 bytes a row and hidden unit with the buffers of every layer
    (3.6 GB for 65,536 rows), 8 with those of one (2.2 GB); 3 GB are left free."""
    n = 65536
    rng = np.random.default_rng(3)
    X = rng.normal(size=(n, 5)).astype(np.float32)
    T = rng.normal(size=(n, 3)).astype(np.float32)
    ref = P.MLP(256, 16, seed=2)
    g0, l0 = ref.grad(X, T)
    h0 = ref.train(X[:999], T[:999], epochs=1, batch=333, lr=1e-3, seed=1)
    p0 = ref.params()
    ref.close()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")
    try:
        mlp = P.MLP(256, 16, seed=2)
        g1, l1 = mlp.grad(X, T)
        h1 = mlp.train(X[:999], T[:999], epochs=1, batch=333, lr=1e-3, seed=1)
        p1 = mlp.params()
        mlp.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    assert l0 == l1 and np.array_equal(g0, g1)
    assert np.array_equal(h0, h1) and np.array_equal(p0, p1)


def test_no_epochs_touch_nothing(lib_path):
    """No copy of X and T is under way when a call of no epochs returns: none is made."""
    n = 1 << 20
    X, T = np.ones((n, 5), np.float32), np.ones((n, 3), np.float32)
    mlp = P.MLP(64, 3, seed=2)
    p = mlp.params()
    free = torch.cuda.mem_get_info()[0]
    assert len(mlp.train(X, T, epochs=0, batch=n, lr=1e-3, seed=1)) == 0
    assert torch.cuda.mem_get_info()[0] == free
    assert np.array_equal(mlp.params(), p)
    mlp.close()
