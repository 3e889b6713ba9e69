"""Launch attributes and occupancy are found per device, by one thread each
(csrc/per_device.cuh)."""
from __future__ import annotations

import subprocess
from pathlib import Path

NATIVE = Path(__file__).resolve().parent / "native"


def test_values_belong_to_a_device(tmp_path):
    exe = tmp_path / "per_device_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-o", str(exe), str(NATIVE / "per_device_check.cpp")],
                   check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
