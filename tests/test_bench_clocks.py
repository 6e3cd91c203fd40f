"""bench.py's clock record: a timed region shorter than nvidia-smi's start has samples of
its own (against a stand-in nvidia-smi, no GPU)."""
import os
import stat
import time

import bench

FAKE = """#!/usr/bin/env python3
import sys, time
time.sleep(0.4)
print("index, clocks.sm [MHz], clocks.max.sm [MHz], ...", flush=True)
lms = float(sys.argv[sys.argv.index("-lms") + 1]) / 1e3
t0 = time.time()
while time.time() - t0 < 20:
    busy = open(sys.argv[0] + ".busy").read()
    print(f"0, {busy} MHz, 1965 MHz, 900 W, 0x0, Not Active, Not Active, Not Active, Active",
          flush=True)
    time.sleep(lms)
"""


def test_a_short_region_is_sampled(tmp_path, monkeypatch):
    smi = tmp_path / "nvidia-smi"
    smi.write_text(FAKE)
    smi.chmod(smi.stat().st_mode | stat.S_IEXEC)
    busy = tmp_path / "nvidia-smi.busy"
    busy.write_text("315")
    monkeypatch.setenv("PATH", f"{tmp_path}{os.pathsep}{os.environ['PATH']}")
    c = bench.ClockSampler(0)
    steps = []
    c.ready(lambda: (steps.append(1), time.sleep(0.01)))
    assert steps                                    # the device is kept busy until then
    busy.write_text("1800")
    time.sleep(0.12)                                # the timed region
    got = c.stop()
    busy.write_text("200")
    assert got["samples"] >= 2 and got["sm_mhz"] == 1800.0 and got["sm_max_mhz"] == 1965.0
    assert got["reasons"] == ["sw_power_cap"]
