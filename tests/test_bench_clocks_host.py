"""The bench's clock record covers a timed region shorter than nvidia-smi's start-up and than its former
sampling period, and holds no sample from before the region."""
import os
import stat
import time

import bench

FAKE = """#!/bin/sh
period=0.2
while [ $# -gt 0 ]; do
  [ "$1" = "-lms" ] && period=$(awk "BEGIN { print $2 / 1000 }")
  shift
done
sleep 0.4
while true; do
  echo "0, 1900, 1965, 500.0, 0x0, Not Active, Not Active, Not Active, Active"
  sleep $period
done
"""


def test_short_region_is_sampled(tmp_path, monkeypatch):
    exe = tmp_path / "nvidia-smi"
    exe.write_text(FAKE)
    exe.chmod(exe.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setenv("PATH", f"{tmp_path}{os.pathsep}{os.environ['PATH']}")
    s = bench.ClockSampler(0)
    s.start()
    s.region()
    t0 = time.monotonic()
    while not s.lines[s.first:] and time.monotonic() < t0 + 5.0:  # a loaded host may be late
        time.sleep(0.15)
    got = s.stop()
    assert (got["sm_mhz"], got["sm_max_mhz"], got["reasons"]) == (1900.0, 1965.0, ["sw_power_cap"]), got
    # none of the time before the region
    assert 1 <= got["samples"] <= (time.monotonic() - t0) / 0.05 + 2, got


def test_without_nvidia_smi(tmp_path, monkeypatch):
    monkeypatch.setenv("PATH", str(tmp_path))
    s = bench.ClockSampler(0)
    s.start()
    assert s.stop()["sm_mhz"] is None
