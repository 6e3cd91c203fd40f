"""A wait of the cluster LU that runs out (a column that is announced to nobody, limit
0.05 s): KLS_ERR_TIMEOUT from every kind of call, and the next call is right again."""
import ctypes as C

import numpy as np
import pytest
import torch

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

BASE = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=11, Ne=5, Rc_min=0.01, Rc_max=10.0,
            v_min=0.01, alpha_max=10.0, l_min=-2, l_max=2, nw=401, nwa=41)
OM = np.array([0.88 + 0.12j, 0.7 + 0.05j])


# one CTA's worth of columns, a ring slot per column, a ring that is used again
@pytest.mark.parametrize("Na", [2, 41, 101, 150])
def test_lu_wait_runs_out(lib_path, Na):
    pc = K.precompute_all(kconfig(**BASE, N_alpha=Na))
    ref = K.compute_determinant_batched(OM, pc)
    call = pc.ctx.call
    call("kls_set_wait_limit", 0.05)

    def timed_out(f):
        call("kls_set_fault_injection", _lib.KLS_FAULT_LU_COLUMN)
        with pytest.raises(_lib.KlsError) as e:
            f()
        assert e.value.code == _lib.KLS_ERR_TIMEOUT, str(e.value)
        assert np.array_equal(K.compute_determinant_batched(OM, pc), ref)

    timed_out(lambda: K.compute_determinant_batched(OM, pc))
    timed_out(lambda: K.set_anchor(pc, OM[0]))
    timed_out(lambda: K.api.ModelBatch([pc], "Float64", batch=2))

    d_om = torch.tensor(OM.view(np.float64), device="cuda")
    d_det = torch.zeros(4, dtype=torch.float64, device="cuda")

    def device():
        call("kls_det_batch_device", C.c_void_p(d_om.data_ptr()), 2, K.KLS_MODE_FP64,
             C.c_void_p(d_det.data_ptr()), C.c_void_p(None))

    torch.cuda.synchronize()
    call("kls_set_fault_injection", _lib.KLS_FAULT_LU_COLUMN)
    device()                                   # does not wait: told by the NaN's bits
    torch.cuda.synchronize()
    assert np.all(d_det.cpu().numpy().view(np.uint64) == 0x7ff8004b4c535455)
    device()
    torch.cuda.synchronize()
    assert np.array_equal(d_det.cpu().numpy(), ref.view(np.float64))
    batch = K.api.ModelBatch([pc], "Float64", batch=2)
    assert np.array_equal(batch.det(OM[None])[0][0], ref)
    batch.close()
    pc.close()
