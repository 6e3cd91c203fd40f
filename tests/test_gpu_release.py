"""kls_release_fp64: what an FP64 batch made before it answers afterwards, and the
device memory that it gives back."""
import numpy as np
import pytest
import torch

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, Ne=21, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            N_alpha=101, alpha_max=10.0, l_min=-10, l_max=10, nw=2001, nwa=101)


@pytest.mark.parametrize("NR", [12, 61])           # over the table / self-similar
def test_fp64_batch_after_a_release(lib_path, NR):
    """The batch's graph holds addresses of the released memory: KLS_ERR_STATE."""
    pcs = [K.precompute_all(kconfig(**GRID, NR=n)) for n in (61, NR)]
    om = np.array([[0.88 + 0.12j, 0.7 + 0.05j]] * 2)
    b64 = K.api.ModelBatch(pcs, "Float64", batch=2)
    b64.det(om)
    K.api.release_fp64(pcs[1])
    for call in (lambda: b64.det(om), lambda: b64.scan(3, 2)):
        with pytest.raises(_lib.KlsError) as e:
            call()
        assert e.value.code == _lib.KLS_ERR_STATE
    b32 = K.api.ModelBatch(pcs, "Float32", batch=2)
    d, _ = b32.det(om)
    assert np.array_equal(d[0], K.compute_determinant_batched(
        om[0], pcs[0], K.to_device(pcs[0], K.GPUType.NVIDIA, "Float32")))
    b32.close()
    b64.close()
    for pc in pcs:
        pc.close()


def test_release_gives_back_the_fp64_buffers(lib_path):
    pc = K.precompute_all(kconfig(**GRID, NR=61))
    K.to_device(pc, K.GPUType.NVIDIA, "Float32")
    K.compute_determinant_batched(np.linspace(0.6, 1.0, 64) + 0.1j, pc)
    rows, Na = 21 * 21, 128                        # F of 64 omegas: 64 bytes a (row, d)
    free = torch.cuda.mem_get_info()[0]
    K.api.release_fp64(pc)
    assert torch.cuda.mem_get_info()[0] - free >= 64 * 64 * rows * Na
    pc.close()
