"""The one-launch time loop of small grids (star7_loop.cuh).

CPU: the numbering of inner and border nodes against plain loops.  GPU: the
loop (inside one cluster on the smallest grids), the sweep by plain loads (star7_march.cuh) and the tile sweeps give the
same bits (an explicitly set depth or tile keeps one launch per step) for every border kind, source, element type and layer count it
accepts, on grids with no inner node, one node, and remainders of warps and
CTAs, over more steps than one launch takes.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

NATIVE = Path(__file__).resolve().parent / "native"


def test_node_numbers_walk_the_grid(tmp_path):
    exe = tmp_path / "node_order_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(NATIVE / "node_order_check.cpp")], check=True)
    grids = [(3, 3, 3, 1), (4, 3, 5, 1), (17, 15, 16, 1), (33, 4, 7, 2), (6, 6, 6, 3), (9, 7, 8, 3), (65, 40, 3, 1)]
    res = subprocess.run([str(exe)] + [str(v) for g in grids for v in g], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


def _problem(M, n, prec, border, source, layers, rng, tile):
    """A handle with every field the problem reads, and its initial iterate."""
    shape = (n[2], n[1], n[0])
    tau = 0.4 / (2.0 * sum((m - 1) ** 2 for m in n))
    kinds = {"dirichlet": M.BORDER_DIRICHLET, "moving": M.BORDER_DIRICHLET, "mirror": M.BORDER_MIRROR_POW2,
             "radiation": M.BORDER_TABLE, "nodes": M.BORDER_NODES, "vc": M.BORDER_DIRICHLET}
    variable = border in ("nodes", "vc")
    heat = dict(c0=1.0, cp=[(m - 1) ** 2 * 1.0 for m in n], cf=1.0) if variable else dict(heat=(1.0, 1.0, 0.3))
    cfg = M.make_cfg(n, tau=tau, t_start=0.25, precision=prec, border=kinds[border], n_layers=layers, tile=tile, **heat)
    p = M.Plain(cfg)
    if source != "none":
        p.upload(M.FIELD_F_A, rng.uniform(0.5, 1.0, shape))
    if source == "affine":
        p.upload(M.FIELD_F_B, rng.uniform(0.5, 1.0, shape))
    if border in ("moving", "radiation"):
        p.upload(M.FIELD_G_A, rng.uniform(0.5, 1.0, shape))
        p.upload(M.FIELD_G_B, rng.uniform(0.5, 1.0, shape))
    if border == "radiation":
        p.set_border_forms(M.border_forms_flux(cfg, M.FLUX_RADIATION, 1.0, 0.1))
        p.set_border_time_basis(0.5, 2.0)
        p.upload(M.FIELD_G_D, rng.uniform(0.0, 0.1, shape))
    if variable:
        p.upload(M.FIELD_C0, rng.uniform(0.2, 0.3, shape))
        p.upload(M.FIELD_CA, tau * rng.uniform(0.5, 1.0, shape))
    if border == "nodes":
        count = M.border_node_count(cfg)
        rules = rng.uniform(0.0, 0.15, (count, 8))
        x, y, z = np.meshgrid(*(np.arange(m) for m in n), indexing="ij")
        at = []
        for axis, m in ((x, n[0]), (y, n[1]), (z, n[2])):
            at += [axis == 0, axis == m - 1]
        border_nodes = np.any(at, axis=0).transpose(2, 1, 0)
        for d in range(6):
            rules[:, 1 + d][at[d].transpose(2, 1, 0)[border_nodes]] = 0.0
        p.set_border_node_rules(rules)
    return p, rng.uniform(0.5, 1.5, shape)


CASES = [(prec, border, source, layers)
         for prec in ("f64", "f32", "f32x2")
         for border, source, layers in (("dirichlet", "none", 1), ("moving", "affine", 1), ("moving", "static", 2),
                                        ("mirror", "static", 1), ("radiation", "static", 1), ("radiation", "affine", 2),
                                        ("nodes", "static", 1), ("nodes", "none", 1), ("vc", "static", 1))
         if prec != "f32x2" or border not in ("nodes", "vc")]


@pytest.mark.gpu
@pytest.mark.parametrize("prec,border,source,layers", CASES)
@pytest.mark.parametrize("n,steps", [((4, 4, 4), 3), ((5, 7, 4), 1030), ((9, 8, 21), 6), ((33, 18, 11), 5), ((70, 66, 68), 4)])
def test_loop_and_sweeps_give_the_same_bits(gpu, prec, border, source, layers, n, steps):
    M = gpu
    got = []
    for schedule in ("loop", "default sweep", "tile"):
        tile = 2 if schedule == "tile" else 0
        p, u0 = _problem(M, n, prec, border, source, layers, np.random.default_rng(n[0] + steps), tile)
        with p:
            if schedule == "default sweep":
                p.set_temporal_depth(1)
            p.upload(M.FIELD_U, u0)
            p.step(1)  # the loop starts at a later step and from the other buffer
            p.step(steps)
            assert p.last_step_launches() == ((steps + 1023) // 1024 if schedule == "loop" else steps)
            assert p.timestep() == steps + 1
            got.append(p.download())
    assert np.all(np.isfinite(got[1])) or border == "mirror"
    assert np.array_equal(got[0], got[1], equal_nan=True)
    assert np.array_equal(got[2], got[1], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32", "f32x2"])
def test_ensemble_schedules_give_the_same_bits(gpu, prec):
    """The ensemble's step by plain loads against the persistent kernel, on
    instances with one inner row, widths around the column tiles' limits and
    a remainder of planes."""
    M = gpu
    rng = np.random.default_rng(4)
    sizes = [(3, 3, 3), (3, 9, 12), (18, 3, 11), (66, 65, 10), (67, 21, 20), (131, 7, 5)]
    specs = [M.batch_instance(n, 0.3 / sum((m - 1) ** 2 for m in n), 0.5, 1.0, 1e-3, 37.0) for n in sizes]
    data = [(37.0 + rng.uniform(0.0, 1.0, n[::-1]), rng.uniform(0.0, 10.0, n[::-1])) for n in sizes]
    got = []
    for tile in (0, 1, 4):
        with M.Batch(specs, prec) as b:
            for i, (u, f) in enumerate(data):
                b.upload(i, M.FIELD_F_A, f)
                b.upload(i, M.FIELD_U, u)
            if tile:
                b.set_schedule(tile)
            else:
                assert b.info()["tile"] == 0
            b.step(5)
            got.append([b.download(i) for i in range(len(sizes))])
    for other in got[1:]:
        for a, c in zip(got[0], other):
            assert np.array_equal(a, c)
