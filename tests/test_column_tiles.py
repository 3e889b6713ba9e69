"""Column tiles of the kernels without a TMA ring (csrc/node_order.cuh).  CPU:
they cover the grid, keep the limits that shared memory is sized by, and are
found in a time that a launch per step can afford on any grid.  GPU: Lame steps
on grids of a few columns, whose CTAs have fewer threads."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

import cases
import oracle as O
from masterthesis_gb300 import workloads as W

NATIVE = Path(__file__).resolve().parent / "native"


def test_column_tiles_cover_the_grid_within_their_limits(tmp_path):
    exe = tmp_path / "column_tile_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(NATIVE / "column_tile_check.cpp")], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(4, 5, 300), (3, 40, 50), (60, 3, 50), (19, 5, 40), (5, 130, 20), (67, 66, 12)])
def test_lame_steps_of_few_columns(gpu, n):
    M = gpu
    T = 8
    rng = np.random.default_rng(n[1])
    shape = (n[2], n[1], n[0])
    u0 = np.zeros((3,) + shape)
    u0[:, 1:-1, 1:-1, 1:-1] = rng.uniform(-1.0, 1.0, u0[:, 1:-1, 1:-1, 1:-1].shape)
    tau = W.lame_tau(n)
    with M.MultiField(M.MF_LAME, n, tau, (1.0, 0.5, 1.0), precision="f64") as mf:
        for c in range(3):
            mf.upload(c, u0[c])
            mf.upload(3 + c, u0[c])
        mf.step(T)
        u = np.stack([mf.download(c) for c in range(3)])
    ref, _ = O.lame(O.make_grid(n, tau=tau), u0, u0, T, 1.0, 0.5, 1.0)
    assert cases.rel_err(u, ref) <= 1e-12
