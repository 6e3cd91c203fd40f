"""The hybrid search on a self-similar model builds no split-BF16 table, which no step of
it reads; an anchored evaluation builds it when it is asked for."""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=61, Ne=21, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            N_alpha=101, alpha_max=10.0, l_min=-10, l_max=10, nw=10001, nwa=201)


def held(pc):
    d = _lib.kls_dims()
    pc.ctx.call("kls_get_dims", d)
    return d.device_bytes, 8 * d.N_alpha_pad * d.K_pad     # hi and lo BF16 of Re and Im


def config():
    c = kconfig(**GRID)
    c.reference.Omega_p, c.reference.gamma = 0.44, 0.12
    c.newton.tol = 1e-12
    return c


def test_hybrid_search_without_the_split_table(lib_path):
    c = config()
    pc, prepared = K.precompute_all(c), K.precompute_all(c)
    K.to_device(prepared, K.GPUType.NVIDIA, "Float32")
    K.compute_determinant_batched([0.9 + 0.1j, 0.9 + 0.11j], pc)      # the FP64 buffers
    before, table = held(pc)
    r = K.api.newton_search_hybrid(c, pc)
    assert held(pc)[0] - before < table
    q = K.api.newton_search_hybrid(c, prepared)
    assert held(prepared)[0] > table
    assert r.converged and (r.Omega_p, r.gamma, r.det_val) == (q.Omega_p, q.gamma, q.det_val)
    assert np.array_equal(r.history, q.history)
    # the anchor, and the evaluation near it that reads the table
    om = 2 * r.Omega_p + 1j * r.gamma
    K.set_anchor(pc, om)
    assert held(pc)[0] - before < table
    dev = K.api.DevicePrecomputed(pc.m, pc.G, pc.N_alpha, pc.n_l, pc.NPh, K.KLS_MODE_ANCHORED, pc)
    K.set_anchor(prepared, om)
    devp = K.api.DevicePrecomputed(pc.m, pc.G, pc.N_alpha, pc.n_l, pc.NPh, K.KLS_MODE_ANCHORED,
                                   prepared)
    near = np.array([om + 1e-6, om + 1e-6j])
    assert np.array_equal(K.compute_determinant_batched(near, pc, dev),
                          K.compute_determinant_batched(near, prepared, devp))
    assert held(pc)[0] - before >= table
    pc.close()
    prepared.close()


def test_hybrid_search_over_the_table_builds_it(lib_path):
    c = config()
    pc = K.precompute_all(c)
    pc.use_table()
    K.compute_determinant_batched([0.9 + 0.1j, 0.9 + 0.11j], pc)
    before, table = held(pc)
    assert K.api.newton_search_hybrid(c, pc).converged
    assert held(pc)[0] - before >= table
    pc.close()
