"""FP64 default schedules bit for bit: the cluster loop, the one-launch loop and
the march (node coefficients too) against C models of the update's operation
order, on fields that keep the integer sums, change sign, tie and span the
exponent range; loops over more steps than one launch takes; one inner node;
and the Lame step against its written-out form."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NATIVE = Path(__file__).resolve().parent / "native"
KINDS = ["smooth", "signed", "ties", "wide"]
dp = C.POINTER(C.c_double)


def _model(tmp_path_factory, name):
    so = tmp_path_factory.mktemp("model") / (name + ".so")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(NATIVE / (name + ".c")),
                    "-lm"], check=True)
    return C.CDLL(str(so))


@pytest.fixture(scope="module")
def star(tmp_path_factory):
    lib = _model(tmp_path_factory, "star7_order")
    lib.star7_sweep_f64.argtypes = [dp, dp, C.c_int, C.c_int, C.c_int] + [C.c_double] * 5
    lib.star7_vc_sweep_f64.argtypes = [dp, dp, dp, dp, C.c_int, C.c_int, C.c_int] + [C.c_double] * 4
    return lib


@pytest.fixture(scope="module")
def lame(tmp_path_factory):
    lib = _model(tmp_path_factory, "lame_order")
    lib.lame_step_f64.argtypes = [dp, dp, dp, C.c_int, C.c_int, C.c_int, dp, dp]
    return lib


def _p(a):
    return a.ctypes.data_as(dp)


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint64)


def _field(kind, shape, rng, span=900.0):
    if kind == "smooth":
        z, y, x = np.meshgrid(*(np.linspace(0.05, 0.95, m) for m in shape), indexing="ij")
        return np.sin(np.pi * x) * np.sin(np.pi * y) * np.sin(np.pi * z) + 1e-3 * rng.random(shape)
    if kind == "signed":
        return rng.uniform(-1.0, 1.0, shape)
    if kind == "ties":  # 53-bit integers: every odd neighbour sum is a rounding tie
        return rng.integers(2 ** 52, 2 ** 53, shape).astype(np.float64)
    v = np.exp2(rng.uniform(-span, span, shape)) * rng.uniform(-2.0, 2.0, shape)
    v[rng.random(shape) < 0.02] = 0.0
    v[rng.random(shape) < 0.02] = -0.0
    sub = rng.random(shape) < 0.02
    v[sub] = 5e-324 * rng.integers(1, 2 ** 40, int(sub.sum()))
    return v


# Cluster loop, one-launch loop, and one launch per step (the march).
PATHS = [((17, 15, 16), "loop"), ((41, 30, 27), "loop"), ((66, 65, 40), "loop"), ((41, 30, 27), "march"),
         ((3, 3, 3), "loop"), ((3, 3, 3), "march")]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,path", PATHS)
@pytest.mark.parametrize("variable", [False, True])
def test_default_steps_equal_the_operation_order_model(gpu, star, kind, n, path, variable):
    M = gpu
    steps = 4
    shape = (n[2], n[1], n[0])
    rng = np.random.default_rng(1 + KINDS.index(kind) + n[0])
    cp = (0.11, 0.09, 0.145)
    c0 = 1.0 if variable else 0.31
    u = np.ascontiguousarray(_field(kind, shape, rng))
    c0f, caf = rng.uniform(0.3, 0.5, shape), rng.uniform(0.6, 1.2, shape)
    with M.Plain(M.make_cfg(n, tau=1e-3, precision="f64", c0=c0, cp=cp, cf=1.0 if variable else 0.0)) as p:
        if variable:
            p.upload(M.FIELD_C0, c0f)
            p.upload(M.FIELD_CA, caf)
        if path == "march":
            p.set_temporal_depth(1)
        p.upload(M.FIELD_U, u)
        p.step(steps)
        assert p.last_step_launches() == (1 if path == "loop" else steps)
        got = p.download()
    for _ in range(steps):
        out = np.empty_like(u)
        if variable:
            star.star7_vc_sweep_f64(_p(u), _p(c0f), _p(caf), _p(out), *n, *cp, 0.0)
        else:
            star.star7_sweep_f64(_p(u), _p(out), *n, c0, *cp, 0.0)
        u = out
    assert np.array_equal(_bits(got), _bits(u))


@pytest.mark.parametrize("prec", ["f64", "f32", "f32x2"])
@pytest.mark.parametrize("border", ["dirichlet", "radiation"])
@pytest.mark.parametrize("steps", [1030, 2049])
def test_loops_of_several_launches_equal_the_sweeps(gpu, prec, border, steps):
    """A grid beyond every cluster limit: the loop over all SMs, whose barrier
    word and step times serve launch after launch."""
    M = gpu
    n = (45, 41, 38)
    shape = (n[2], n[1], n[0])
    tau = 0.4 / (2.0 * sum((m - 1) ** 2 for m in n))
    table = border == "radiation"
    cfg = M.make_cfg(n, tau=tau, t_start=0.25, precision=prec, border=M.BORDER_TABLE if table else M.BORDER_DIRICHLET,
                     heat=(1.0, 1.0, 0.3))
    got = []
    for loop in (True, False):
        rng = np.random.default_rng(steps)
        with M.Plain(cfg) as p:
            if table:
                p.set_border_forms(M.border_forms_flux(cfg, M.FLUX_RADIATION, 1.0, 0.1))
            for slot in (M.FIELD_F_A, M.FIELD_F_B, M.FIELD_G_A, M.FIELD_G_B):
                p.upload(slot, rng.uniform(0.5, 1.0, shape))
            if not loop:
                p.set_temporal_depth(1)
            p.upload(M.FIELD_U, rng.uniform(0.5, 1.5, shape))
            p.step(1)
            p.step(steps)
            assert p.last_step_launches() == ((steps + 1023) // 1024 if loop else steps)
            got.append(p.download())
    assert np.all(np.isfinite(got[0])) and np.array_equal(got[0], got[1])


@pytest.mark.parametrize("kind", ["smooth", "signed", "ties", "wide"])
@pytest.mark.parametrize("n", [(3, 3, 3), (18, 7, 20), (67, 19, 13), (131, 9, 11)])
def test_lame_step_equals_the_written_out_form(gpu, lame, kind, n):
    M = gpu
    steps = 3
    shape = (n[2], n[1], n[0])
    rng = np.random.default_rng(n[0])
    lam, mu, rho, tau = 1.0, 0.5, 1.25, 0.2 / max(n)
    hh = [1.0 / (m - 1) for m in n]
    s = tau * tau / rho
    a = np.array([[s * (lam + 2.0 * mu if p == c else mu) / (hh[p] * hh[p]) for p in range(3)] for c in range(3)])
    b = np.array([[0.0 if p == c else s * (lam + mu) / (4.0 * hh[c] * hh[p]) for p in range(3)] for c in range(3)])
    now = np.stack([_field(kind, shape, rng, 250.0) for _ in range(3)])
    before = np.stack([_field(kind, shape, rng, 250.0) for _ in range(3)])
    with M.MultiField(M.MF_LAME, n, tau, (lam, mu, rho), precision="f64") as mf:
        for c in range(3):
            mf.upload(c, now[c])
            mf.upload(3 + c, before[c])
        mf.step(steps)
        got = np.stack([mf.download(c) for c in range(3)])
    for _ in range(steps):
        out = np.empty_like(now)
        lame.lame_step_f64(_p(now), _p(before), _p(out), *n, _p(a), _p(b))
        now, before = out, now
    assert np.array_equal(_bits(got), _bits(now))
