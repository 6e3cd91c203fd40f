"""Grids beyond the launch limits of the self-similar form: they are evaluated over the
table, and a split count above the limit is clamped.  Against the sum over every
orbit's own W on the host, each entry within the rounding of the two sums (K terms):
2 (K + 8) 2^-53 of the sum of moduli, and the accepted misfit of an orbit (1.01e-10 of
its amplitude) where the self-similar form runs."""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

BASE = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            N_alpha=2, alpha_max=5.0, nw=401, nwa=41)


def close_to_host_sum(pc, M, om):
    W = pc.W_l_mat.transpose(2, 0, 1).reshape(-1, pc.N_alpha)
    w = (pc.DJ_vec[:, None] * pc.F0l_all / (om - pc.Omega_res)).T.reshape(-1)
    GN = pc.G * pc.N_kernel[None, :]
    ref = GN * (W.T @ (w[:, None] * W.conj()))
    g = pc.orbit_data.grids
    amp = np.tile((1.0 / np.sqrt(g.Rc * (1.0 - g.e))).reshape(-1, order="F"), len(w) // pc.NPh)
    tol = np.abs(GN) * (2 * (len(w) + 8) * 2.0 ** -53 * (np.abs(W).T @ (np.abs(w)[:, None] * np.abs(W)))
                        + 2 * 1.01e-10 * np.sum(np.abs(w) * amp ** 2))
    return np.all(np.abs(M - ref) <= tol)


@pytest.mark.parametrize("NR,Ne,nl", [(16, 65535, 17), (16, 65537, 1), (131073, 2, 1)])
def test_grids_beyond_the_launch_limits(lib_path, NR, Ne, nl):
    lo = -(nl // 2)
    pc = K.precompute_all(kconfig(**BASE, NR=NR, Ne=Ne, l_min=lo, l_max=lo + nl - 1))
    om = 0.88 + 0.12j
    assert close_to_host_sum(pc, K.build_M_matrix(om, pc), om)
    pc.close()


def test_split_count_beyond_the_launch_limit(lib_path):
    """270,000 rows (l, e) allow 33,750 splits of 8 rows: two CTA rows each, 67,500."""
    pc = K.precompute_all(kconfig(**BASE, NR=16, Ne=30000, l_min=-4, l_max=4))
    pc.ctx.call("kls_set_splits", K.KLS_MODE_FP64, 10 ** 6)
    om = 0.88 + 0.12j
    assert close_to_host_sum(pc, K.build_M_matrix(om, pc), om)
    pc.close()
