"""Copies to the device are ordered with the kernels that read them.

The library's streams are non-blocking, so they do not wait for the default stream.
A synchronous copy from pageable memory may return before its data is on the device,
and one between device buffers, like a memset, always may: none of them may be used
for what a kernel reads next.  (A race cannot be made to fail by running it.)"""
import glob
import os
import re

from tests.conftest import ROOT


def test_no_unordered_copies_to_the_device():
    bad = []
    for p in glob.glob(os.path.join(ROOT, "kalnajs_log_spirals_b200", "csrc", "*.cu")):
        src = open(p).read()
        for m in re.finditer(r"\bcuda(Memcpy|Memset)\(", src):
            end = src.index(";", m.start())
            if m.group(1) == "Memset" or "DeviceToHost" not in src[m.start():end]:
                bad.append((os.path.basename(p), src[m.start():end]))
    assert not bad, bad
