"""The pipelined LU at the edges of its size classes (rows per lane, columns per
warp, ring slots) against the one-CTA LU: same pivots, same operations in the
same order on every element, hence the same bits; and against LAPACK on the
host, det(I - M) within 2 N^2 2^-53 relative of numpy's (backward error of both
factorisations, times the condition of these diagonally dominant matrices).
"""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

BASE = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=11, Ne=5, Rc_min=0.01, Rc_max=10.0,
            v_min=0.01, alpha_max=10.0, l_min=-2, l_max=2, nw=401, nwa=41)


@pytest.mark.parametrize("Na", [1, 2, 7, 8, 9, 31, 32, 33, 62, 63, 64, 65, 96, 101, 127, 128, 129,
                                160, 191, 192, 193, 224, 255, 256, 257, 301, 320, 321, 400, 512])
def test_pipelined_lu_is_bitwise_the_cta_lu(lib_path, Na):
    pc = K.precompute_all(kconfig(**BASE, N_alpha=Na))
    rng = np.random.default_rng(Na)
    om = 2 * rng.uniform(0.3, 0.6, 20) + 1j * rng.uniform(0.02, 0.25, 20)
    out = []
    for mode in (_lib.KLS_LU_CTA, _lib.KLS_LU_CLUSTER, _lib.KLS_LU_AUTO):
        pc.ctx.call("kls_set_lu_mode", mode)
        out.append(K.compute_determinant_batched(om, pc, None, batch_size=16, log_abs=True))
    M = K.build_M_matrix(om[0], pc)
    pc.close()
    for d, la in out[1:]:
        assert np.array_equal(d, out[0][0]), np.max(np.abs(d - out[0][0]) / np.abs(out[0][0]))
        assert np.array_equal(la, out[0][1])
    ref = np.linalg.det(np.eye(Na) - M)
    cond = np.linalg.cond(np.eye(Na) - M)
    assert abs(out[0][0][0] - ref) <= 2 * Na ** 2 * 2.0 ** -53 * cond * abs(ref)


@pytest.mark.parametrize("Na", [225, 240, 416, 417])
def test_pipelined_lu_between_classes(lib_path, Na):
    """Further edges of the classes, at batches of 16 (the class's form) and 2 (its
    wider one where it has one): the bits of the one-CTA LU."""
    pc = K.precompute_all(kconfig(**BASE, N_alpha=Na))
    rng = np.random.default_rng(Na)
    om = 2 * rng.uniform(0.3, 0.6, 18) + 1j * rng.uniform(0.02, 0.25, 18)
    out = []
    for mode in (_lib.KLS_LU_CTA, _lib.KLS_LU_AUTO):
        pc.ctx.call("kls_set_lu_mode", mode)
        out.append(K.compute_determinant_batched(om, pc, None, batch_size=16, log_abs=True))
    pc.close()
    assert np.array_equal(out[1][0], out[0][0])
    assert np.array_equal(out[1][1], out[0][1])
