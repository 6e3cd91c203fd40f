"""kls_autotune's cache: a model's FP64 split count is not another's of the same padded
sizes whose count means something else (row splits of the pair sum on self-similar
orbits, K splits over the table) or is limited otherwise."""
import pytest

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, v_min=0.01, alpha_max=10.0, nw=2001, nwa=101)
# (NR, Ne, l_max, N_alpha, Rc_min): K = 840 terms, padded to 896, N_alpha to 64
TABLE = (24, 5, 3, 33, 1e-7)                  # orbits below the integrator's thresholds
OTHERS = [(24, 5, 3, 33, 0.01),               # the same sizes, self-similar
          (24, 5, 3, 63, 0.01), (40, 3, 3, 33, 0.01), (24, 7, 2, 33, 0.01)]


def tune(size):
    NR, Ne, lm, Na, rmin = size
    pc = K.precompute_all(kconfig(**GRID, NR=NR, Ne=Ne, l_min=-lm, l_max=lm, N_alpha=Na, Rc_min=rmin,
                                  Rc_max=1.0))
    t = K.api.autotune(pc, "Float64", batch=3)
    pc.close()
    return t


def test_each_model_is_tuned_for_itself(lib_path):
    for size in [TABLE] + OTHERS:
        first = tune(size)
        assert first.candidates >= 1, size
        again = tune(size)
        assert again.candidates == 0 and again.splits == first.splits, size
