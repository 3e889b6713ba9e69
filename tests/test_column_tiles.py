"""Column tiles of the kernels without a TMA ring (csrc/node_order.cuh):
they cover the grid, keep the limits that shared memory is sized by, and are
found in a time that a launch per step can afford on any grid."""
from __future__ import annotations

import subprocess
from pathlib import Path

NATIVE = Path(__file__).resolve().parent / "native"


def test_column_tiles_cover_the_grid_within_their_limits(tmp_path):
    exe = tmp_path / "column_tile_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(NATIVE / "column_tile_check.cpp")], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
