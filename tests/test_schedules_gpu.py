"""What the schedules choose on the GPU: the autotuner's choice is what later
steps run, the defaults are near the best schedule, loops of several handles
overlap.  Times are compared between schedules of the same problem, measured
one after the other, best of several; the margins are far below what a wrong
choice costs, and a comparison that a disturbance spoils is made again."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def heat(M, n, prec, tile=0, seed=1, source="none", layers=1):
    rng = np.random.default_rng(seed)
    shape = (n[2], n[1], n[0])
    tau = 0.4 / (2.0 * sum((m - 1) ** 2 for m in n))
    p = M.Plain(M.make_cfg(n, tau=tau, precision=prec, n_layers=layers, tile=tile, heat=(1.0, 1.0, 0.3)))
    if source != "none":
        p.upload(M.FIELD_F_A, rng.uniform(0.5, 1.0, shape))
    if source == "affine":
        p.upload(M.FIELD_F_B, rng.uniform(0.5, 1.0, shape))
    p.upload(M.FIELD_U, rng.uniform(0.5, 1.5, shape))
    return p


def us_per_step(p, steps=60):
    """Best of four step calls, by the device's clock."""
    best = np.inf
    for _ in range(4):
        p.step(steps)
        p.synchronize()
        best = min(best, p.last_step_ms())
    return 1e3 * best / steps


def assert_no_slower(margin, measure, tries=4):
    """measure() -> (time, time of what it is compared with)."""
    for _ in range(tries):
        t, reference = measure()
        if t <= margin * reference:
            return
    assert t <= margin * reference


@pytest.mark.parametrize("prec", ["f64", "f32", "f32x2"])
@pytest.mark.parametrize("n", [(17, 15, 16), (64, 48, 40), (160, 160, 160)])
def test_autotuned_steps_run_what_was_fastest(gpu, prec, n):
    M = gpu
    with heat(M, n, prec) as p:

        def measure():  # a second call chooses anew
            _, ms = p.autotune(20)
            t = us_per_step(p)
            launches = p.last_step_launches()
            assert launches == 30 if p.temporal_depth == 2 else launches in (1, 60)
            return t, 1e3 * min(ms)

        assert_no_slower(1.15, measure)
        assert_no_slower(1.15, measure)


def test_autotune_keeps_one_launch_per_step_of_a_set_tile(gpu):
    M = gpu
    with heat(M, (17, 15, 16), "f64", tile=2) as p:
        p.autotune(5)
        p.step(8)
        assert p.last_step_launches() in (4, 8)


@pytest.mark.parametrize("instances,side", [(5, 94), (8, 90), (10, 90), (13, 95)])
def test_default_pair_ensemble_schedule_is_near_the_best(gpu, instances, side):
    M = gpu
    rng = np.random.default_rng(instances)
    n = (side + 3, side, side - 3)
    shape = (n[2], n[1], n[0])
    tau = 0.3 / sum((m - 1) ** 2 for m in n)
    with M.Batch([M.batch_instance(n, tau, 0.5, 1.0, 1e-3, 37.0)] * instances, "f32x2") as b:
        for i in range(instances):
            b.upload(i, M.FIELD_F_A, rng.uniform(0.0, 10.0, shape))
            b.upload(i, M.FIELD_U, 37.0 + rng.uniform(0.0, 1.0, shape))

        def best(tile):
            if tile is not None:
                b.set_schedule(tile)
            ms = []
            for _ in range(4):
                b.step(30)
                ms.append(b.last_ms())
            return min(ms)

        chosen = b.info()["tile"]
        assert_no_slower(1.12, lambda: (best(chosen), min(best(tile) for tile in (1, 2, 3, 4))))


@pytest.mark.parametrize("prec,source,layers,n", [
    ("f32x2", "affine", 1, (150, 140, 145)), ("f32x2", "affine", 1, (260, 258, 120)), ("f32x2", "static", 1, (140, 150, 145)),
    ("f32x2", "static", 2, (240, 230, 220)), ("f32", "none", 2, (224, 220, 200)), ("f32", "static", 2, (150, 140, 145)),
    ("f32", "affine", 2, (201, 181, 163)), ("f32x2", "none", 2, (130, 129, 131)), ("f32", "none", 1, (100, 100, 300)),
    ("f32", "none", 1, (130, 130, 5)), ("f32", "affine", 1, (200, 200, 20)), ("f32x2", "none", 1, (64, 64, 1000))])
def test_default_sweep_is_near_the_best(gpu, prec, source, layers, n):
    M = gpu

    def measure():
        us = []
        for tile in (0, 1, 2, 3, 4):
            with heat(M, n, prec, tile, source=source, layers=layers) as p:
                p.set_temporal_depth(1)
                us.append(us_per_step(p))
        return us[0], min(us[1:])

    assert_no_slower(1.12, measure)


@pytest.mark.parametrize("prec,source,n", [("f32", "none", (160, 160, 160)), ("f32", "none", (250, 240, 230)),
                                           ("f32", "static", (201, 181, 163)), ("f32x2", "affine", (130, 140, 120)),
                                           ("f64", "static", (201, 181, 163)), ("f64", "none", (80, 80, 80))])
def test_default_steps_are_near_the_faster_of_loop_and_sweeps(gpu, prec, source, n):
    M = gpu

    def measure():
        with heat(M, n, prec, source=source) as p:
            default = us_per_step(p)
            p.set_temporal_depth(1)
            return default, us_per_step(p)

    assert_no_slower(1.1, measure)


@pytest.mark.parametrize("prec", ["f64", "f32", "f32x2"])
@pytest.mark.parametrize("n", [(50, 50, 50), (64, 64, 64)])
def test_loops_of_several_handles_share_the_gpu(gpu, prec, n):
    """Four handles on streams of their own: their loops overlap (in turn they
    would take four times as long as one), and give the bits of loops run
    alone."""
    M = gpu
    steps = 400
    handles = [heat(M, n, prec, seed=k) for k in range(4)]

    def seconds(some):
        best = np.inf
        for _ in range(3):
            for p in some:
                p.synchronize()
            t0 = time.perf_counter()
            for p in some:
                p.step(steps)
            for p in some:
                p.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best

    try:
        alone = []
        for k in range(4):
            with heat(M, n, prec, seed=k) as p:
                p.step(steps)
                assert p.last_step_launches() == 1
                alone.append(p.download())
        for p in handles:
            p.step(steps)
        for p, want in zip(handles, alone):
            assert np.array_equal(p.download(), want)
        assert_no_slower(3.2, lambda: (seconds(handles), seconds(handles[:1])))
    finally:
        for p in handles:
            p.close()


@pytest.mark.parametrize("prec,side", [("f64", 20), ("f32", 20), ("f32", 170)])
def test_a_reported_ensemble_schedule_can_be_set_again(gpu, prec, side):
    M = gpu
    n = (side, side, side)
    tau = 0.3 / (3.0 * (side - 1) ** 2)
    u0 = np.random.default_rng(side).uniform(37.0, 38.0, n)
    got = []
    for again in (False, True):
        with M.Batch([M.batch_instance(n, tau, 0.5, 1.0, 0.0, 37.0)], prec) as b:
            b.upload(0, M.FIELD_U, u0)
            b.step(2)
            info = b.info()
            if again:
                b.set_schedule(2)
                b.step(2)
                b.set_schedule(info["tile"], info["ctas_per_sm"])
                assert {k: b.info()[k] for k in ("tile", "ctas_per_sm", "items")} == \
                    {k: info[k] for k in ("tile", "ctas_per_sm", "items")}
                b.step(2)
            else:
                b.step(4)
            got.append(b.download(0))
    assert np.array_equal(got[0], got[1])
    with M.Batch([M.batch_instance(n, tau, 0.5, 1.0, 0.0, 37.0)], prec) as b:
        for tile in (-1, 5):
            with pytest.raises(M.ScafesError):
                b.set_schedule(tile)
