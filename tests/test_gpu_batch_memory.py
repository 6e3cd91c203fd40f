"""A large FP64 batch over self-similar models holds the pair sums' partials of one range
of omegas of one model at a time, and its determinants are each model's own."""
import numpy as np
import pytest
import torch

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=20, Ne=21, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            alpha_max=10.0, l_min=-25, l_max=25, nw=2001, nwa=101)


def test_partials_of_a_large_batch(lib_path):
    """1071 rows (l, e), N_alpha 33: 17 MB of partials an omega, 1 GB (61 omegas) at a
    time; 150 omegas, one range for both models, 256 MB of F and 0.1 GB of weights and
    matrices beside it."""
    pcs = [K.precompute_all(kconfig(**GRID, N_alpha=n)) for n in (33, 31)]
    om = np.linspace(0.6, 1.0, 150) + 0.1j
    assert all(pc.self_similar for pc in pcs)
    ref = [K.compute_determinant_batched(om, pc) for pc in pcs]
    M = [K.build_M_matrix(om[0], pc) for pc in pcs]
    free = torch.cuda.mem_get_info()[0]
    mb = K.api.ModelBatch(pcs, "Float64", batch=150)
    assert free - torch.cuda.mem_get_info()[0] <= 1.6e9
    d, _ = mb.det(np.stack([om, om]))
    mb.close()
    assert np.array_equal(d, ref)
    # and one model's own calls at a split count whose partials pass the limit
    pcs[0].ctx.call("kls_set_splits", K.KLS_MODE_FP64, 60)
    few = K.compute_determinant_batched(om[:40], pcs[0])
    assert np.array_equal(few[:3], K.compute_determinant_batched(om[:3], pcs[0]))
    assert np.max(np.abs(few - ref[0][:40]) / np.abs(ref[0][:40])) <= 1e-11
    assert np.array_equal(M[1], K.build_M_matrix(om[0], pcs[1]))
    for pc in pcs:
        pc.close()
