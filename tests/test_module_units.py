"""What the first determinant of a process loads.  A module (one translation unit's device
code) is loaded as a whole at the first call that needs a kernel of it, 0.5 ms a megabyte:
each size class of the pipelined LU is a unit of its own, and the weights, which every
form takes, are not in the unit of the table's contraction."""
import glob
import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "kalnajs_log_spirals_b200", "csrc")


def source(name):
    return open(os.path.join(CSRC, name)).read()


def test_one_lu_class_a_unit():
    classes = re.findall(r"\blup_kernels_(\d+)\b", source("kls_lu_pipe.h"))
    units = {os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "kls_lu_*.cu"))}
    assert classes and units == {f"kls_lu_{n}.cu" for n in classes}
    for n in classes:
        assert re.findall(r"LUP_DEFINE\((\d+),", source(f"kls_lu_{n}.cu")) == [n]
    assert "kls_lu_pipe.cuh\"" not in source("kls_lu.cu")


def test_weights_apart_from_the_contraction():
    assert "void weights_kernel(" in source("kls_basis.cu")
    assert not re.search(r"__global__[^;{]*weights_kernel\(", source("kls_contract.cu"))
