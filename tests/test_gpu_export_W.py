"""kls_export_W: a harmonic has the same bits however it is asked for (alone, in any block,
over the table or from the samples), and W(-alpha) = conj W(alpha)."""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            alpha_max=10.0, nw=401, nwa=41)


@pytest.mark.parametrize("Na,NR,Ne,l", [(1, 16, 3, 3), (2, 17, 3, 20), (33, 33, 5, 9), (64, 31, 2, 17),
                                        (101, 16, 7, 5)])
def test_bits_of_a_harmonic(lib_path, Na, NR, Ne, l):
    pc = K.precompute_all(kconfig(**GRID, N_alpha=Na, NR=NR, Ne=Ne, l_min=-l, l_max=l + 1))
    W = pc.W_l_mat
    nl = 2 * l + 2
    assert W.shape == (NR * Ne, Na, nl)
    assert Na == 1 or np.array_equal(W, W[:, ::-1].conj())     # (one alpha is -alpha_max)
    for il in range(nl):
        assert np.array_equal(pc.export_W(il, 1)[..., 0], W[..., il]), il
    for il, n in ((1, nl - 1), (3, 2), (nl - 2, 2), (0, 0), (2, nl - 3)):
        assert np.array_equal(pc.export_W(il, n), W[..., il:il + n])
    assert pc.self_similar
    pc.use_table()
    assert np.array_equal(pc.W_l_mat, W)
    assert np.array_equal(pc.export_W(nl - 1, 1)[..., 0], W[..., -1])
    pc.close()


def test_ranges_of_alpha(lib_path):
    """More than 32 MB a harmonic: its alphas go in ranges; and blocks of harmonics."""
    pc = K.precompute_all(kconfig(**GRID, N_alpha=151, NR=400, Ne=35, l_min=-1, l_max=3))
    W = pc.W_l_mat
    pc.use_table()
    assert np.array_equal(pc.W_l_mat, W) and np.array_equal(W, W[:, ::-1].conj())
    one = pc.export_W(2, 1)
    assert np.array_equal(one[..., 0], W[..., 2]) and np.abs(W).min(axis=(0, 1)).max() > 0
    pc.close()
