"""M(omega) from the self-similar orbits (csrc/kls_similar.cu) at the edges of
its tiles, against the sum over every orbit's own W on the host:
    G N(a) sum_k W[k, b] w_k conj(W[k, a]),   w_k = DJ F0l / (omega - Omega_res).

Tolerance per entry, derived: rounding of the two sums, 2 (K + 8) 2^-53 of the
sum of moduli; and the accepted misfit of an orbit, 1e-10 (its samples) + 1e-12
(second order) of its amplitude |W| <= (Rc (1 - e))^-1/2, in both factors.
N_alpha runs over the 32 x 32 pair tiles' edges, even and odd; NR over the 16
radii a slab holds; the row splits over one, a few and the most allowed.
"""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            alpha_max=10.0, nw=2001, nwa=101)


def launches(pc):
    return pc.ctx.lib.kls_launch_count(pc.ctx.h)


@pytest.mark.parametrize("Na,NR,Ne,l", [(1, 16, 2, 1), (2, 16, 3, 2), (31, 17, 5, 3), (32, 16, 5, 3),
                                        (33, 40, 4, 2), (63, 33, 3, 3), (64, 32, 5, 4),
                                        (65, 31, 5, 2), (97, 48, 7, 3), (101, 61, 6, 4),
                                        (128, 20, 4, 3), (150, 37, 5, 5), (301, 16, 3, 2)])
def test_matrix_against_every_orbit(lib_path, Na, NR, Ne, l):
    pc = K.precompute_all(kconfig(**GRID, N_alpha=Na, NR=NR, Ne=Ne, l_min=-l, l_max=l + 1))
    om = 0.88 + 0.12j
    W = pc.W_l_mat.transpose(2, 0, 1).reshape(-1, Na)
    w = (pc.DJ_vec[:, None] * pc.F0l_all / (om - pc.Omega_res)).T.reshape(-1)
    GN = np.abs(pc.G * pc.N_kernel[None, :])
    ref = pc.G * pc.N_kernel[None, :] * (W.T @ (w[:, None] * W.conj()))
    g = pc.orbit_data.grids
    amp = np.tile((1.0 / np.sqrt(g.Rc * (1.0 - g.e))).reshape(-1, order="F"), W.shape[0] // pc.NPh)
    tol = GN * (2 * (len(w) + 8) * 2.0 ** -53 * (np.abs(W).T @ (np.abs(w)[:, None] * np.abs(W)))
                + 2 * 1.01e-10 * np.sum(np.abs(w) * amp ** 2))
    try:
        for splits in (None, 1, 3, 10 ** 6):
            if splits:
                pc.ctx.call("kls_set_splits", K.KLS_MODE_FP64, splits)
            n0 = launches(pc)
            M = K.build_M_matrix(om, pc)
            # weights, F, pair sum, reduction (and the determinant stage)
            assert launches(pc) - n0 >= 4
            assert np.all(np.abs(M - ref) <= tol), (Na, splits, np.max(np.abs(M - ref) / tol))
            d = K.compute_determinant_batched(np.array([om, 0.7 + 0.05j, om]), pc)
            assert d[0] == d[2] == K.compute_determinant(om, pc)
    finally:
        pc.close()


def test_orbits_of_another_form_keep_the_table(lib_path):
    """Radii so small that L^2 falls below the integrator's thresholds (1e-12,
    1e-14) for some of a column's orbits: no common form, the sum runs over the
    table and equals the host's (rounding bound as above)."""
    c = dict(GRID, Rc_min=1e-7, Rc_max=1.0)
    pc = K.precompute_all(kconfig(**c, N_alpha=33, NR=24, Ne=5, l_min=-2, l_max=2))
    om = 0.88 + 0.12j
    W = pc.W_l_mat.transpose(2, 0, 1).reshape(-1, 33)
    w = (pc.DJ_vec[:, None] * pc.F0l_all / (om - pc.Omega_res)).T.reshape(-1)
    GN = pc.G * pc.N_kernel[None, :]
    M = K.build_M_matrix(om, pc)
    pc.close()
    tol = np.abs(GN) * 2 * (len(w) + 8) * 2.0 ** -53 * (np.abs(W).T @ (np.abs(w)[:, None] * np.abs(W)))
    assert np.all(np.abs(M - GN * (W.T @ (w[:, None] * W.conj()))) <= tol)
