"""A call that ran out of device memory says so, and the next one is right again: the
failed allocation's error is not left for its launch check."""
import numpy as np
import pytest
import torch

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib, proposer as P
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu


@pytest.fixture
def little_memory(lib_path):
    """200 MB of the device left free."""
    torch.cuda.empty_cache()
    fill = []
    yield lambda: fill.append(torch.empty(torch.cuda.mem_get_info()[0] - (200 << 20),
                                          dtype=torch.uint8, device="cuda"))
    fill.clear()
    torch.cuda.empty_cache()


def refused(f, code):
    with pytest.raises(_lib.KlsError) as e:
        f()
    assert e.value.code == code, str(e.value)


def test_determinants_after_out_of_memory(little_memory):
    c = kconfig(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=200, Ne=30, Rc_min=0.01, Rc_max=10.0,
                v_min=0.01, N_alpha=201, alpha_max=20.0, l_min=-40, l_max=40, nw=2001, nwa=101)
    om = np.linspace(0.6, 1.0, 16) + 0.1j
    pc = K.precompute_all(c)
    ref = K.compute_determinant_batched(om[:2], pc)
    M = K.build_M_matrix(om[0], pc)
    little_memory()
    refused(lambda: K.compute_determinant_batched(om, pc), _lib.KLS_ERR_OOM)
    assert np.array_equal(K.compute_determinant_batched(om[:1], pc), ref[:1])
    refused(lambda: K.to_device(pc, K.GPUType.NVIDIA, "Float32"), _lib.KLS_ERR_OOM)
    assert np.array_equal(K.build_M_matrix(om[0], pc), M)
    refused(pc.use_table, _lib.KLS_ERR_OOM)
    assert pc.self_similar and np.array_equal(K.compute_determinant_batched(om[:2], pc), ref)
    refused(lambda: K.api.ModelBatch([pc], "Float64", batch=64), _lib.KLS_ERR_OOM)
    assert np.array_equal(K.compute_determinant_batched(om[:2], pc), ref)
    refused(lambda: K.precompute_all(kconfig(**dict(
        m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=900, Ne=30, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
        N_alpha=301, alpha_max=20.0, l_min=-60, l_max=60, nw=2001, nwa=1001))), _lib.KLS_ERR_OOM)
    assert np.array_equal(K.compute_determinant_batched(om[:2], pc), ref)
    pc.close()


def test_proposer_after_out_of_memory(little_memory):
    rng = np.random.default_rng(1)
    X = rng.normal(size=(1 << 17, 5)).astype(np.float32)
    T = rng.normal(size=(1 << 17, 3)).astype(np.float32)
    mlp = P.MLP(256, 4, seed=3)
    ref = mlp.forward(X[:100])
    little_memory()
    refused(lambda: mlp.grad(X, T), _lib.KLS_ERR_CUDA)
    assert np.array_equal(mlp.forward(X[:100]), ref)
    other = P.MLP(256, 4, seed=3)
    assert np.array_equal(other.params(), mlp.params())
    other.close()
    mlp.close()
