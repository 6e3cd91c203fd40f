"""The split-BF16 form's output rows at the edges of its MMA widths: N_alpha rounded
up to 32 where one MMA takes all rows (up to 256), else to 64.  Against plain FP64:
the split form's error is a few 1e-5 of the determinant (a row that is not formed
would be an error of order one), and the batch of two models runs the same body.
"""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

BASE = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=41, Ne=11, Rc_min=0.01, Rc_max=10.0,
            v_min=0.01, alpha_max=10.0, l_min=-4, l_max=4, nw=2001, nwa=201)


@pytest.mark.parametrize("Na", [33, 64, 65, 95, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225,
                                256, 257, 320])
def test_split_form_against_fp64(lib_path, Na):
    c = kconfig(**BASE, N_alpha=Na)
    pc = K.precompute_all(c)
    om = np.array([0.9 + 0.2j, 0.8 + 0.1j, 1.0 + 0.05j])
    ref = K.compute_determinant_batched(om, pc, None)
    M = K.build_M_matrix(om[0], pc)
    dev = K.to_device(pc, K.GPUType.NVIDIA, "Float32")
    pc.ctx.call("kls_set_mixed_form", _lib.KLS_MIXED_TMEM)
    d = K.compute_determinant_batched(om, pc, dev)
    Mx = K.build_M_matrix(om[0], pc, dev)
    batch = K.ModelBatch([pc], "Float32", batch=3)
    db, _ = batch.det(om[None])
    batch.close()
    pc.close()
    assert np.max(np.abs(Mx - M)) <= 1e-4 * np.max(np.abs(M))
    assert np.all(np.abs(d - ref) <= 1e-3 * np.abs(ref))
    assert np.array_equal(db[0], d)
