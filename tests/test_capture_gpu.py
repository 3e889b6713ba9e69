"""A step call while another stream of the program is being captured into a
CUDA graph (global mode): the first call of a fresh handle must not make an
allocation, which the runtime refuses then, spoiling the capture as well."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32", "f32x2"])
@pytest.mark.parametrize("border", ["dirichlet", "radiation"])
@pytest.mark.parametrize("n", [(9, 8, 7), (40, 31, 27), (66, 70, 64)])
def test_first_steps_during_a_capture_elsewhere(gpu, prec, border, n):
    M = gpu
    rt = C.CDLL("libcudart.so.13")
    tau = 0.4 / (2.0 * sum((m - 1) ** 2 for m in n))
    shape = (n[2], n[1], n[0])
    rng = np.random.default_rng(2)
    u0, f, g = (rng.uniform(0.5, 1.5, shape) for _ in range(3))
    table = border == "radiation"
    cfg = M.make_cfg(n, tau=tau, precision=prec, border=M.BORDER_TABLE if table else M.BORDER_DIRICHLET,
                     heat=(1.0, 1.0, 0.3))
    got = []
    for captured in (False, True):
        with M.Plain(cfg) as p:
            if table:
                p.set_border_forms(M.border_forms_flux(cfg, M.FLUX_RADIATION, 1.0, 0.1))
                p.upload(M.FIELD_F_A, f)
                p.upload(M.FIELD_G_A, g)
            p.upload(M.FIELD_U, u0)
            stream, graph = C.c_void_p(), C.c_void_p()
            if captured:
                assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
                assert rt.cudaStreamBeginCapture(stream, 0) == 0
            try:
                p.step(10)
            finally:
                if captured:
                    end = rt.cudaStreamEndCapture(stream, C.byref(graph))
                    if graph:
                        rt.cudaGraphDestroy(graph)
                    rt.cudaStreamDestroy(stream)
                    rt.cudaGetLastError()
            if captured:
                assert end == 0
            got.append(p.download())
    assert np.array_equal(got[0], got[1])
