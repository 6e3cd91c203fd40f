"""smoke() runs the FP64 path that most models take, F and the pair sums over the common
orbits, and the table's contraction beside it."""
import re

import pytest

import __graft_entry__ as entry
import kalnajs_log_spirals_b200 as K

pytestmark = pytest.mark.gpu


def test_smoke_runs_both_fp64_forms(lib_path, monkeypatch, capsys):
    forms = []
    plain = K.compute_determinant_batched

    def noted(om, pc, dev=None, **kw):
        if dev is None:
            forms.append(pc.ctx.lib.kls_get_f64_similar(pc.ctx.h))
        return plain(om, pc, dev, **kw)

    monkeypatch.setattr(K, "compute_determinant_batched", noted)
    entry.smoke()
    assert {0, 1} <= set(forms), forms
    assert re.search(r"smoke: det rel err", capsys.readouterr().out)
