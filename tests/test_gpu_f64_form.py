"""Which FP64 form a model takes, shown by the query and by the launches, and the choice of
the table by the caller."""
import numpy as np
import pytest

import kalnajs_log_spirals_b200 as K
from kalnajs_log_spirals_b200 import _lib
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, v_min=0.01, alpha_max=10.0, nw=2001, nwa=101)
SIMILAR = dict(Rc_min=0.01, Rc_max=10.0)
# radii so small that L^2 falls below the integrator's thresholds for some orbits
OTHER = dict(Rc_min=1e-7, Rc_max=1.0)
OM = np.array([0.88 + 0.12j, 0.7 + 0.05j, 1.1 + 0.2j])


def launches_of_M(pc):
    n0 = pc.ctx.lib.kls_launch_count(pc.ctx.h)
    M = K.build_M_matrix(OM[0], pc)
    return pc.ctx.lib.kls_launch_count(pc.ctx.h) - n0, M


def tolerance(pc, M):
    """Of an entry of M between the two forms: the rounding of either sum over the K terms
    and the accepted misfit of an orbit (1.01e-10 of its amplitude), as for the sum over
    every orbit."""
    W = pc.W_l_mat.transpose(2, 0, 1).reshape(-1, pc.N_alpha)
    w = np.abs((pc.DJ_vec[:, None] * pc.F0l_all / (OM[0] - pc.Omega_res)).T.reshape(-1))
    g = pc.orbit_data.grids
    amp = np.tile((1.0 / np.sqrt(g.Rc * (1.0 - g.e))).reshape(-1, order="F"), len(w) // pc.NPh)
    return np.abs(pc.G * pc.N_kernel[None, :]) * (
        2 * (len(w) + 8) * 2.0 ** -53 * (np.abs(W).T @ (w[:, None] * np.abs(W)))
        + 2 * 1.01e-10 * np.sum(w * amp ** 2))


@pytest.mark.parametrize("Na,NR,Ne,l", [(1, 16, 2, 1), (2, 16, 3, 2), (33, 40, 4, 2),
                                        (65, 31, 5, 2), (101, 61, 6, 4), (150, 37, 5, 5)])
def test_self_similar_and_by_choice_the_table(lib_path, Na, NR, Ne, l):
    pc = K.precompute_all(kconfig(**GRID, **SIMILAR, N_alpha=Na, NR=NR, Ne=Ne, l_min=-l, l_max=l))
    assert pc.self_similar
    n, M = launches_of_M(pc)
    assert n == 5                      # weights, F, pair sum, reduction, transpose
    d = K.compute_determinant_batched(OM, pc)
    tol = tolerance(pc, M)
    batch = K.api.ModelBatch([pc], "Float64", batch=3)
    pc.use_table()
    assert not pc.self_similar
    nt, Mt = launches_of_M(pc)
    assert nt == 4                     # weights, contraction, reduction, transpose
    assert np.all(np.abs(M - Mt) <= tol)
    dt = K.compute_determinant_batched(OM, pc)
    # a batch made before keeps its form, one made now takes the table until it is freed
    assert np.array_equal(batch.det(OM[None])[0][0], d)
    over_table = K.api.ModelBatch([pc], "Float64", batch=3)
    assert np.array_equal(over_table.det(OM[None])[0][0], dt)
    pc.use_table(False)
    assert pc.self_similar and launches_of_M(pc)[0] == 5
    assert np.array_equal(K.compute_determinant_batched(OM, pc), d)
    assert np.array_equal(batch.det(OM[None])[0][0], d)
    with pytest.raises(_lib.KlsError) as e:
        over_table.det(OM[None])
    assert e.value.code == _lib.KLS_ERR_STATE
    batch.close()
    over_table.close()
    pc.close()


BASE = dict(GRID, **SIMILAR, N_alpha=65, NR=40, Ne=9, l_min=-6, l_max=7)


@pytest.mark.parametrize("options", [
    dict(m=0), dict(m=-2), dict(m=5), dict(n_zang=0), dict(q1=1.2), dict(q1=40),
    dict(v_min=-1.0), dict(v_min=-0.9, Ne=7), dict(v_min=0.995, Ne=5), dict(Ne=1),
    dict(Rc_min=1.0, Rc_max=1.0), dict(Rc_min=1e-4, Rc_max=1e4, NR=101), dict(alpha_max=0.0),
    dict(alpha_max=300.0, N_alpha=129), dict(L0=1e-3), dict(G=1e6), dict(l_min=5, l_max=9),
    dict(l_min=0, l_max=0), dict(nw=401, nwa=9), dict(nw=101, nwa=101),
    dict(quadrature="sss"), dict(quadrature="bbb", NR=41), dict(quadrature="tst", NR=41)])
def test_forms_agree_over_the_options(lib_path, options):
    """Harmonic number, disk, retrograde and radial orbits, equal radii, a single alpha or
    eccentricity, quadratures: where the model is self-similar, M as over the table."""
    o = dict(BASE, **options)
    quadrature = o.pop("quadrature", "tts")
    c = kconfig(**o)
    c.grid.quadrature = quadrature
    pc = K.precompute_all(c)
    assert pc.self_similar
    with np.errstate(all="ignore"):
        M = K.build_M_matrix(OM[0], pc)
        tol = tolerance(pc, M)
        pc.use_table()
        assert np.all(np.abs(M - K.build_M_matrix(OM[0], pc)) <= tol)
    pc.close()


@pytest.mark.parametrize("grid,NR", [(SIMILAR, 15), (OTHER, 24)])
def test_models_over_the_table(lib_path, grid, NR):
    """Fewer than 16 radii, or orbits of another form."""
    pc = K.precompute_all(kconfig(**GRID, **grid, N_alpha=33, NR=NR, Ne=5, l_min=-2, l_max=2))
    assert not pc.self_similar and launches_of_M(pc)[0] == 4
    d = K.compute_determinant_batched(OM, pc)
    for on in (True, False):           # nothing to choose
        pc.use_table(on)
        assert not pc.self_similar
        assert np.array_equal(K.compute_determinant_batched(OM, pc), d)
    K.api.release_fp64(pc)
    assert pc.ctx.lib.kls_get_f64_similar(pc.ctx.h) == -1
    with pytest.raises(_lib.KlsError) as e:
        pc.use_table()
    assert e.value.code == _lib.KLS_ERR_STATE
    pc.close()
