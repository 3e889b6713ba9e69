"""Signs of zeros: the integer adder's (CPU, bit for bit against the host's
FP64 adder), and those of a Yee step and of recorded linear rules on fields of
zeros of both signs, where every operation is exact and numpy gives the bits."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

NATIVE = Path(__file__).resolve().parent / "native"


@pytest.mark.parametrize("seed", [7, 19])
def test_any_sign_adder_gives_the_fp64_adders_bits(tmp_path, seed):
    exe = tmp_path / "dadd_any_bits_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(NATIVE / "dadd_any_bits_check.cpp")], check=True)
    res = subprocess.run([str(exe), str(seed), "4000000"], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


def bits(a):
    return np.ascontiguousarray(a).view(np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(5, 4, 6), (35, 7, 9)])
def test_yee_step_of_signed_zeros(gpu, n):
    M = gpu
    rng = np.random.default_rng(n[0])
    shape = (n[2], n[1], n[0])
    f = [np.where(rng.random(shape) < 0.5, -0.0, 0.0) for _ in range(6)]
    tau = 0.25 / (n[0] - 1)
    ch = tau * (n[0] - 1)
    src = (1, 1, 1)
    with M.MultiField(M.MF_YEE, n, tau, (0.0, 0.0, 1.0, 1.0), precision="f64", src=src) as mf:
        for i, a in enumerate(f):
            mf.upload(i, a)
        mf.step(1)
        got = [mf.download(i) for i in range(6)]
    ex, ey, ez, hx, hy, hz = (a.copy() for a in f)
    up, lo = slice(1, None), slice(None, -1)
    hx[lo, lo, :] = -ch * ((ez[lo, up, :] - ez[lo, lo, :]) - (ey[up, lo, :] - ey[lo, lo, :])) + hx[lo, lo, :]
    hy[lo, :, lo] = -ch * ((ex[up, :, lo] - ex[lo, :, lo]) - (ez[lo, :, up] - ez[lo, :, lo])) + hy[lo, :, lo]
    hz[:, lo, lo] = -ch * ((ey[:, lo, up] - ey[:, lo, lo]) - (ex[:, up, lo] - ex[:, lo, lo])) + hz[:, lo, lo]
    i, d = slice(1, -1), slice(None, -2)
    ex[i, i, lo] = ch * ((hz[i, i, lo] - hz[i, d, lo]) - (hy[i, i, lo] - hy[d, i, lo])) + ex[i, i, lo]
    ey[i, lo, i] = ch * ((hx[i, lo, i] - hx[d, lo, i]) - (hz[i, lo, i] - hz[i, lo, d])) + ey[i, lo, i]
    ez[lo, i, i] = ch * ((hy[lo, i, i] - hy[lo, i, d]) - (hx[lo, i, i] - hx[lo, d, i])) + ez[lo, i, i]
    at = (src[2], src[1], src[0])  # the source's own zero joins in here
    got[2][at] = ez[at] = 0.0
    for k, want in enumerate((ex, ey, ez, hx, hy, hz)):
        assert np.array_equal(bits(got[k]), bits(want)), k


@pytest.mark.gpu
@pytest.mark.parametrize("cst", [0.0, -0.0])
def test_linear_rules_of_signed_zeros(gpu, cst):
    """A rule is a chain of fma from its constant on: a copy of -0 with the
    constant +0 gives +0, with -0 it stays."""
    M = gpu
    n = (6, 5, 4)
    shape = (n[2], n[1], n[0])
    rng = np.random.default_rng(3)
    f = [np.where(rng.random(shape) < 0.5, -0.0, 0.0) for _ in range(2)]
    with M.Linear(n, 2) as h:
        for cls in range(64):
            h.set_rule(1, 0, cls, [(1, 0, 0, 0, 1.0)], cst)
            h.set_rule(1, 1, cls, [(0, 0, 0, 0, 1.0), (1, 0, 0, 0, 0.5)], cst)
        for i, a in enumerate(f):
            h.upload(i, a)
        h.step(1)
        got = [h.download(i) for i in range(2)]
    want = [f[1] + cst, 0.5 * f[1] + (f[0] + cst)]
    for a, b in zip(got, want):
        assert np.array_equal(bits(a), bits(b))
