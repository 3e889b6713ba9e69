"""Grids of 2^31 nodes and more, which the dense 32-bit node numbers do not
cover: the Yee step's second slab of planes, and the column form of the Lame
step.  The fields are zero but for the last
planes; those are compared with numpy (FP64: a few roundings of numbers of
order one).  Needs 130 GB on the device and 40 GB on the host."""
from __future__ import annotations

import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (1300, 1300, 1275)  # 2.15e9 nodes; slabs of 1270 planes
SHAPE = N[::-1]
Z0 = 1262               # the fields' first nonzero plane
TOL = 1e-14
up, lo, inner, below = slice(1, None), slice(None, -1), slice(1, -1), slice(None, -2)


@pytest.fixture(scope="module")
def room(gpu):
    free, total = C.c_size_t(), C.c_size_t()
    assert C.CDLL("libcudart.so.13").cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
    if free.value < 150e9 or os.sysconf("SC_PAGE_SIZE") * os.sysconf("SC_AVPHYS_PAGES") < 60e9:
        pytest.skip("not enough memory for 2^31 nodes")
    return gpu


def _last(seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, (SHAPE[0] - Z0,) + SHAPE[1:])


def _field(seed):
    a = np.zeros(SHAPE)
    a[Z0:] = _last(seed)
    return a


def _end(seed):
    """Planes Z0 - 2 and on of the field."""
    return np.concatenate([np.zeros((2,) + SHAPE[1:]), _last(seed)])


def _check(h, field, want):
    got = h.download(field)
    assert np.abs(got[Z0 + 1:] - want[3:]).max() <= TOL * np.abs(want[3:]).max()
    assert not np.any(got[5:Z0 - 4:97, ::61, ::61])


def test_yee_step_in_slabs(room):
    M = room
    tau = 0.25 / (N[0] - 1)
    ch = tau * (N[0] - 1)
    with M.MultiField(M.MF_YEE, N, tau, (0.0, 0.0, 1.0, 1.0), "f64", src=(5, 5, 5)) as h:
        for i in range(6):
            h.upload(i, _field(i))
        h.step(1)
        ex, ey, ez, hx, hy, hz = (_end(i) for i in range(6))
        hx[lo, lo, :] -= ch * ((ez[lo, up, :] - ez[lo, lo, :]) - (ey[up, lo, :] - ey[lo, lo, :]))
        hy[lo, :, lo] -= ch * ((ex[up, :, lo] - ex[lo, :, lo]) - (ez[lo, :, up] - ez[lo, :, lo]))
        hz[:, lo, lo] -= ch * ((ey[:, lo, up] - ey[:, lo, lo]) - (ex[:, up, lo] - ex[:, lo, lo]))
        i, d = inner, below
        ex[i, i, lo] += ch * ((hz[i, i, lo] - hz[i, d, lo]) - (hy[i, i, lo] - hy[d, i, lo]))
        ez[lo, i, i] += ch * ((hy[lo, i, i] - hy[lo, i, d]) - (hx[lo, i, i] - hx[lo, d, i]))
        for f, want in ((0, ex), (2, ez), (3, hx), (5, hz)):
            _check(h, f, want)


def test_lame_step_by_columns(room):
    M = room
    tau, lam, mu, rho = 0.1 / N[0], 1.0, 0.5, 1.0
    hh = [1.0 / (m - 1) for m in N]
    s = tau * tau / rho
    with M.MultiField(M.MF_LAME, N, tau, (lam, mu, rho), "f64") as h:
        for i in range(6):
            h.upload(i, _field(i))
        h.step(1)
        u = [_end(i) for i in range(3)]

        def at(a, **move):
            cut = []
            for axis, m in zip("zyx", a.shape):
                k = move.get(axis, 0)
                cut.append(slice(1 + k, m - 1 + k))
            return a[tuple(cut)]

        for c in (0, 2):
            acc = 2.0 * at(u[c]) - at(_end(3 + c))
            for p in range(3):
                a = s * (lam + 2.0 * mu if p == c else mu) / hh[p] ** 2
                acc += a * (at(u[c], **{"xyz"[p]: 1}) + at(u[c], **{"xyz"[p]: -1}) - 2.0 * at(u[c]))
            for q in range(3):
                if q == c:
                    continue
                d = [at(u[q], **{"xyz"[c]: i, "xyz"[q]: j}) for i in (1, -1) for j in (1, -1)]
                acc += s * (lam + mu) / (4.0 * hh[c] * hh[q]) * ((d[0] - d[1]) - (d[2] - d[3]))
            want = np.zeros_like(u[c])
            want[inner, inner, inner] = acc
            _check(h, c, want)
