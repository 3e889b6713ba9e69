"""The barrier of the one-launch time loop is bounded: it gives up on CTAs that
never arrive, sets the status word, and leaves the context usable."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu

TIMEOUT = -6


@pytest.mark.parametrize("limit_us", [20000, 200000])
def test_grid_barrier_gives_up_and_reports(gpu, limit_us):
    M = gpu
    fn = M.lib().scafes_probe_grid_barrier_timeout
    fn.argtypes = [C.c_uint, C.POINTER(C.c_int), C.POINTER(C.c_double)]
    st, ms = C.c_int(), C.c_double()
    assert fn(0, C.byref(st), C.byref(ms)) == -1
    assert fn(limit_us, C.byref(st), C.byref(ms)) == 0
    assert st.value == TIMEOUT
    # after the limit, and within 256 polls of it (some hundred us)
    assert limit_us / 1000.0 <= ms.value <= limit_us / 1000.0 + 50.0
    n, T = (41, 30, 27), 10
    u0 = np.random.default_rng(1).uniform(-1.0, 1.0, (n[2], n[1], n[0]))
    tau = 0.9 / (2.0 * sum((m - 1) ** 2 for m in n))
    with M.Plain(M.make_cfg(n, tau=tau, heat=(1.0, 1.0, 0.0))) as p:
        p.upload(M.FIELD_U, u0)
        p.step(T)
        assert p.last_step_launches() == 1
        assert cases.rel_err(p.download(), O.heat_dirichlet(O.make_grid(n, tau=tau), u0, T)) <= 1e-12
