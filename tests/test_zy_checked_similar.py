"""The bounds-checked build covers the self-similar FP64 form: every kernel of it is
guarded, and at shapes that take it no access is skipped (tests/checked_similar_run.py,
in a fresh process that binds libkls_checked.so)."""
import os
import re
import subprocess
import sys

import pytest

from tests.conftest import ROOT


def test_every_kernel_is_guarded():
    src = open(os.path.join(ROOT, "kalnajs_log_spirals_b200", "csrc", "kls_similar.cu")).read()
    parts = re.split(r"^__global__", src, flags=re.M)[1:]
    assert len(parts) >= 10
    for p in parts:
        body = p[:re.search(r"^}", p, flags=re.M).start()]
        assert "SIM_IN(" in body or "SIM_AT(" in body, body[:60]


@pytest.mark.gpu
def test_checked_similar_form(lib_path):
    from kalnajs_log_spirals_b200 import build
    build.build(checked=True)                  # no-op when libkls_checked.so is current
    out = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "checked_similar_run.py")],
                         capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert out.returncode == 0 and "CHECKED_OK" in out.stdout, out.stdout + out.stderr[-3000:]
