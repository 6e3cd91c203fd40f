"""The FP64 contraction at the edges of its 8 x 8 blocks and 64 x 64 parts.

M(omega) against the reference's own sum over the library's exported tables,
    G N(a) sum_k W[k, b] w_k conj(W[k, a]),   w_k = DJ F0l / (omega - Omega_res),
in FP64 on the host.  Both sides sum K terms in FP64, so each entry may be off
by at most 2 (K + 8) 2^-53 G N(a) sum_k |W[k, b]| |w_k| |W[k, a]| (K - 1
additions and a handful of products per term, each within 2^-53 of its partial
sum's bound, on either side).  N_alpha runs over one block, one group, a part
with 1 to 8 block rows, and even counts (no alpha = 0); the split counts over
one item per part, a few and the most the table allows.
"""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, NR=11, Ne=5, Rc_min=0.01, Rc_max=10.0,
            v_min=0.01, alpha_max=10.0, l_min=-3, l_max=4, nw=401, nwa=41)


def reference(pc, omega):
    W = pc.W_l_mat.transpose(2, 0, 1).reshape(-1, pc.N_alpha)          # [K, N_alpha]
    w = (pc.DJ_vec[:, None] * pc.F0l_all / (omega - pc.Omega_res)).T.reshape(-1)
    M = W.T @ (w[:, None] * W.conj())
    bound = np.abs(W).T @ (np.abs(w)[:, None] * np.abs(W))
    GN = pc.G * pc.N_kernel[None, :]
    return GN * M, 2 * (len(w) + 8) * 2.0 ** -53 * np.abs(GN) * bound


@pytest.mark.parametrize("Na", [1, 2, 7, 8, 9, 17, 41, 56, 57, 63, 64, 65, 66, 74, 81, 90, 97,
                                105, 113, 121, 128, 129, 150, 193])
def test_matrix_at_tile_edges(lib_path, Na):
    pc = K.precompute_all(kconfig(**GRID, N_alpha=Na))
    om = 0.88 + 0.12j
    ref, tol = reference(pc, om)
    try:
        for splits in (None, 1, 2, 7, 10 ** 6):
            if splits:
                pc.ctx.call("kls_set_splits", K.KLS_MODE_FP64, splits)
            M = K.build_M_matrix(om, pc)
            assert np.all(np.abs(M - ref) <= tol), (Na, splits, np.max(np.abs(M - ref) / tol))
    finally:
        pc.close()
