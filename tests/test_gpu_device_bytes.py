"""kls_get_dims.device_bytes is the device memory that the context holds: the common orbits'
arrays are in it, and a buffer that is grown or given back counts once or not at all."""
import numpy as np
import pytest
import torch

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu


def held(pc):
    d = _lib.kls_dims()
    pc.ctx.call("kls_get_dims", d)
    return d.device_bytes


def test_device_bytes_follow_the_memory(lib_path):
    """Against the driver's figure, to the 2 MB pages (at most 20 allocations) and 8 MB of
    code that first launches load."""
    c = kconfig(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=200, Ne=30, Rc_min=0.01, Rc_max=10.0,
                v_min=0.01, N_alpha=301, alpha_max=30.0, l_min=-40, l_max=40, nw=2001, nwa=101)
    om = np.linspace(0.6, 1.0, 16) + 0.1j
    warm = K.precompute_all(c)
    K.compute_determinant_batched(om, warm)
    warm.close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    used = lambda: free - torch.cuda.mem_get_info()[0]
    slack = 20 * (2 << 20) + (8 << 20)
    pc = K.precompute_all(c)
    rows, half = 30 * 81, 304                      # What, FP32 What and D: 20 bytes a value
    assert held(pc) >= 20 * rows * half + 24 * 101 * 200 * 30
    assert abs(held(pc) - used()) <= slack
    for n in (1, 3, 16):
        K.compute_determinant_batched(om[:n], pc)
        assert abs(held(pc) - used()) <= slack, n
    pc.close()
