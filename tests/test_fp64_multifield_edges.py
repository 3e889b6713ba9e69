"""FP64 Yee and Lame steps whose sums run partly on the integer pipe.

CPU: the any-sign integer adder against the host's FP64 adder.  GPU: one Yee
step on fields that keep the integer path (smooth), change sign everywhere,
span exponents far apart, or hold zeros (the FP64 fallback), against the same
formula in numpy within the bound of its roundings; the Lame step on grids
that cut its column tiles and plane chunks every way, against the oracle.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

import cases
import oracle as O
from masterthesis_gb300 import workloads as W

NATIVE = Path(__file__).resolve().parent / "native"


@pytest.mark.parametrize("seed", [3, 11])
def test_any_sign_adder_equals_the_fp64_adder(tmp_path, seed):
    exe = tmp_path / "dadd_any_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(NATIVE / "dadd_any_check.cpp")], check=True)
    res = subprocess.run([str(exe), str(seed), "4000000"], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    pairs, handed_back = map(int, res.stdout.split())
    assert handed_back < pairs // 3


@pytest.mark.parametrize("seed", [5, 13])
def test_constant_factor_multiplier_equals_the_fp64_multiplier(tmp_path, seed):
    exe = tmp_path / "dmul_int_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(NATIVE / "dmul_int_check.cpp")], check=True)
    res = subprocess.run([str(exe), str(seed), "4000000"], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


def _field(kind, shape, rng):
    if kind == "smooth":
        z, y, x = np.meshgrid(*(np.linspace(0.1, 0.9, m) for m in shape), indexing="ij")
        return 1.0 + x + y * z + 1e-3 * rng.random(shape)
    u = rng.uniform(-1.0, 1.0, shape)
    if kind == "wide":
        u *= np.exp2(rng.integers(-300, 300, shape).astype(np.float64))
    if kind == "zeros":
        u[rng.random(shape) < 0.3] = 0.0
        u[rng.random(shape) < 0.1] *= 1e-310
    return u


def _diff(v, a, b, d, e, c):
    """v + c ((a - b) - (d - e)) and the sum of its terms' magnitudes."""
    return v + c * ((a - b) - (d - e)), np.abs(v) + abs(c) * (np.abs(a) + np.abs(b) + np.abs(d) + np.abs(e))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["smooth", "signed", "wide", "zeros"])
@pytest.mark.parametrize("n", [(3, 3, 3), (33, 6, 5), (70, 9, 8)])
def test_yee_step_within_its_roundings(gpu, kind, n):
    M = gpu
    rng = np.random.default_rng(len(kind) + n[0])
    shape = (n[2], n[1], n[0])
    f = [_field(kind, shape, rng) for _ in range(6)]
    tau = 0.5 / (n[0] - 1) / np.sqrt(3.0)
    ch = tau * (n[0] - 1)
    with M.MultiField(M.MF_YEE, n, tau, (0.0, 0.0, 1.0, 1.0), precision="f64", src=(1, 1, 1)) as mf:
        for i, a in enumerate(f):
            mf.upload(i, a)
        mf.step(1)
        got = [mf.download(i) for i in range(6)]
    ex, ey, ez, hx, hy, hz = (a.copy() for a in f)
    s = np.s_
    # Each update has four roundings here (the products c * (...) round once
    # more in numpy): 8 half-ulps of the sum of its terms' magnitudes cover
    # both sides.  The E step's bound adds its H values' bounds.
    eps = 8 * 2.0 ** -53
    bound = [np.zeros(shape) for _ in range(6)]
    lo, up = s[:-1], s[1:]

    al = s[:]
    for t, h, (a, da), (d, dd) in ((3, hx, (ez, "y"), (ey, "z")), (4, hy, (ex, "z"), (ez, "x")),
                                   (5, hz, (ey, "x"), (ex, "y"))):
        axes = {"z": (lo if "z" in (da, dd) else al), "y": (lo if "y" in (da, dd) else al),
                "x": (lo if "x" in (da, dd) else al)}
        base = (axes["z"], axes["y"], axes["x"])

        def moved(k):
            return tuple(up if ax == k else sl for ax, sl in zip("zyx", base))

        v, mag = _diff(h[base], a[moved(da)], a[base], d[moved(dd)], d[base], -ch)
        h[base] = v
        bound[t][base] = eps * mag
    inner = s[1:-1]
    for t, e, own, (a, da), (d, dd) in ((0, ex, "x", (hz, "y"), (hy, "z")), (1, ey, "y", (hx, "z"), (hz, "x")),
                                        (2, ez, "z", (hy, "x"), (hx, "y"))):
        base = tuple(lo if ax == own else inner for ax in "zyx")

        def below(k):
            return tuple(s[:-2] if ax == k else sl for ax, sl in zip("zyx", base))

        v, mag = _diff(e[base], a[base], a[below(da)], d[base], d[below(dd)], ch)
        e[base] = v
        ba, bd = (bound[3 + next(k for k, m in enumerate((hx, hy, hz)) if m is f)] for f in (a, d))
        bound[t][base] = eps * mag + ch * (ba[base] + ba[below(da)] + bd[base] + bd[below(dd)])
    for i, want in enumerate((ex, ey, ez, hx, hy, hz)):
        assert np.all(np.abs(got[i] - want) <= bound[i] + 1e-320), (kind, i)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(3, 3, 3), (12, 40, 5), (18, 7, 20), (67, 19, 13), (131, 5, 9)])
def test_lame_step_on_cut_tiles(gpu, n):
    M = gpu
    T = 12
    u0 = W.gaussian_bump_displacement(n, seed=5)
    rng = np.random.default_rng(n[0])
    u0[:, 1:-1, 1:-1, 1:-1] += 1e-3 * rng.uniform(-1.0, 1.0, u0[:, 1:-1, 1:-1, 1:-1].shape)
    tau = W.lame_tau(n)
    with M.MultiField(M.MF_LAME, n, tau, (1.0, 0.5, 1.0), precision="f64") as mf:
        for c in range(3):
            mf.upload(c, u0[c])
            mf.upload(3 + c, u0[c])
        mf.step(T)
        u = np.stack([mf.download(c) for c in range(3)])
    ref, _ = O.lame(O.make_grid(n, tau=tau), u0, u0, T, 1.0, 0.5, 1.0)
    assert cases.rel_err(u, ref) <= 1e-12
