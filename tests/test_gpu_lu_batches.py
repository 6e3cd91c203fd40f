"""Uneven batches on both sides of the LU's rule between a cluster per matrix and one CTA
per matrix: the bits of each model's own determinants."""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

BASE = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=11, Ne=3, Rc_min=0.01, Rc_max=10.0,
            v_min=0.01, alpha_max=10.0, l_min=-2, l_max=2, nw=401, nwa=41)


@pytest.mark.parametrize("Tgpu,Nas", [("Float64", (41,)), ("Float64", (101, 128)),
                                      ("Float64", (150, 101)), ("Float32", (150, 41))])
@pytest.mark.parametrize("batch", [8, 100, 310])
def test_batch_on_either_side(lib_path, Tgpu, Nas, batch):
    pcs = [K.precompute_all(kconfig(**BASE, N_alpha=Na)) for Na in Nas]
    om = np.linspace(0.6, 1.0, batch) + 0.1j
    mb = K.api.ModelBatch(pcs, Tgpu, batch=batch)
    d, la = mb.det(np.stack([om] * len(Nas)))
    mb.close()
    for pc, di, li in zip(pcs, d, la):
        pc.ctx.call("kls_set_lu_mode", _lib.KLS_LU_CTA)
        dev = K.to_device(pc, K.GPUType.NVIDIA, Tgpu)
        ref, lref = K.compute_determinant_batched(om, pc, dev, log_abs=True)
        assert np.array_equal(di, ref) and np.array_equal(li, lref)
        pc.close()
