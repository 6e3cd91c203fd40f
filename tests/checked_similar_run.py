"""Run the self-similar FP64 form on libkls_checked.so (run as a script).

As checked_build_run.py, at shapes that take this form (16 radii and more; odd and even
numbers of radii and of alphas, one and several tiles of pairs, ragged rows): every
determinant within 1e-11 of the oracle's, M within 1e-11 of its largest entry, and no
skipped access.  Prints CHECKED_OK and exits 0 when all of that holds.
"""
import ctypes as C
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

from kalnajs_log_spirals_b200 import _lib  # noqa: E402

LIB = _lib.load(_lib.CHECKED_LIB_PATH)     # before any other load: the API runs on it

import kalnajs_log_spirals_b200 as K  # noqa: E402
from oracle import np_oracle as O  # noqa: E402
from tests.test_gpu_parity import kconfig  # noqa: E402

BASE = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            alpha_max=10.0, nw=1001, nwa=101)
# (NR, Ne, N_alpha, l_max)
SHAPES = [(16, 2, 1, 1), (17, 5, 33, 3), (40, 3, 64, 2), (33, 7, 97, 4)]


def main() -> int:
    ok = True
    om = np.array([0.88 + 0.12j, 0.7 + 0.05j, 1.1 + 0.2j])
    for NR, Ne, Na, l in SHAPES:
        over = dict(BASE, NR=NR, Ne=Ne, N_alpha=Na, l_min=-l, l_max=l)
        pc = K.precompute_all(kconfig(**over), device=0)
        similar = pc.self_similar
        d = K.compute_determinant_batched(om, pc)
        M = K.build_M_matrix(om[0], pc)
        pc.ctx.call("kls_set_splits", K.KLS_MODE_FP64, 3)
        d3 = K.compute_determinant_batched(om, pc)
        pc.close()
        opc = O.precompute_all(O.OracleConfig(**over))
        do = np.array([O.compute_det(opc, w) for w in om])
        Mo = O.build_M(opc, om[0])
        e = max(float(np.max(np.abs(x - do) / np.abs(do))) for x in (d, d3))
        eM, top = float(np.max(np.abs(M - Mo))), float(np.max(np.abs(Mo)))   # (0 at N_alpha = 1)
        v, site, idx, ext = C.c_int64(), C.c_int32(), C.c_int64(), C.c_int64()
        code = LIB.kls_bounds_report(C.byref(v), C.byref(site), C.byref(idx), C.byref(ext), 1)
        print(f"{NR} x {Ne}, N_alpha {Na}: self-similar {similar}, report code {code} violations "
              f"{v.value} (site {site.value}, index {idx.value}, extent {ext.value}); det {e:.2e}, "
              f"M {eM:.2e} of {top:.2e}", flush=True)
        ok = ok and similar and code == 0 and v.value == 0 and e <= 1e-11 and eM <= 1e-11 * top
    print("CHECKED_OK" if ok else "CHECKED_FAIL", flush=True)
    return 0 if ok else 1


if __name__ == "__main__":
    sys.exit(main())
