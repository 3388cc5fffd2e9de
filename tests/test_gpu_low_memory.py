"""Solves whose buffers do not fit beside the default kernel run in a form that needs less memory,
with the same times; the next solve takes the default again."""
import numpy as np
import pytest

from conftest import random_slowness

pytestmark = pytest.mark.gpu

import eikonalxx_gb300 as ex  # noqa: E402

GRID = nx, ny, nz = 41, 34, 30


def _bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


def _run(solve, opt):
    """(times, launches): the default, with the first attempt taken not to fit, and the default again."""
    c, f = solve
    out = []
    for fail in (0, 1, 0):
        t = f(ex.Options(**opt, test_alloc_fail=fail))
        out.append(([np.array(q) for q in t], c.stats()["kernel_launches"]))
    return out


def _check(out, lean_launches):
    for t, _ in out[1:]:
        for a, b in zip(t, out[0][0]):
            assert np.array_equal(_bits(a), _bits(b))
    assert out[0][1] == out[2][1]
    if lean_launches is not None:
        assert out[1][1] == lean_launches != out[0][1]


@pytest.mark.parametrize("precision,near", [(ex.F32, False), (ex.F32, True), (ex.F64, False)])
@pytest.mark.parametrize("spacing", [(50.0, 50.0, 50.0), (50.0, 65.0, 40.0)])
@pytest.mark.parametrize("form", ["plain", "pairs asked for", "warm", "stream"])
def test_3d_falls_back_to_the_chunk_step_kernel(ctx, form, spacing, precision, near):
    rng = np.random.default_rng(91)
    dt = np.float32 if precision == ex.F32 else np.float64
    ctx.set_grid3d(*GRID, *spacing)
    ctx.set_slowness3d(random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=dt))
    pos = rng.uniform(0, 1, (6, 3)) * (np.array(GRID) - 1) * spacing
    opt = dict(n_sweeps=3, tolerance=1e-5, near_fp64=near)
    if form == "warm":
        init = ctx.solve3d(pos, ex.Options(**opt), precision) * dt(1.02)
        f = lambda o: ctx.solve3d_warm(pos, init, o, precision)
    else:
        f = lambda o: ctx.solve3d(pos, o, precision)
    if form == "stream":
        opt["max_in_flight"] = 2   # one ordering per launch in either kernel
    f(ex.Options(**opt, sweep_kernel=2))
    chunk = ctx.stats()["kernel_launches"]
    if form == "pairs asked for":
        opt["pair_fields"] = True
    out = _run((ctx, f), opt)
    _check(out, None if form in ("stream", "pairs asked for") else chunk)


@pytest.mark.parametrize("precision", [ex.F32, ex.F64])
def test_a_batch_falls_back(ctx, precision):
    rng = np.random.default_rng(92)
    dt = np.float32 if precision == ex.F32 else np.float64
    models = []
    for g in ((23, 17, 12, 100.0, 100.0, 100.0), (14, 11, 16, 60.0, 80.0, 70.0), (40, 12, 19, 50.0, 50.0, 50.0)):
        models.append({"grid": g, "model": random_slowness(rng, (g[2] - 1) * (g[1] - 1) * (g[0] - 1), dtype=dt),
                       "sources": [(120.0, 130.0, 140.0), (300.0, 400.0, 500.0)]})
    opt = dict(n_sweeps=3, tolerance=1e-5)
    ctx.solve3d_batch(models, ex.Options(**opt, sweep_kernel=2), precision)
    chunk = ctx.stats()["kernel_launches"]
    _check(_run((ctx, lambda o: ctx.solve3d_batch(models, o, precision)), opt), chunk)


@pytest.mark.parametrize("precision", [ex.F32, ex.F64])
@pytest.mark.parametrize("spacing", [(10.0, 10.0), (10.0, 12.5)])
def test_2d_falls_back_to_one_ordering_per_launch(ctx, spacing, precision):
    rng = np.random.default_rng(93)
    dt = np.float32 if precision == ex.F32 else np.float64
    ctx.set_grid2d(61, 70, *spacing)
    ctx.set_slowness2d(random_slowness(rng, 60 * 69, dtype=dt))
    pos = rng.uniform(0, 1, (5, 2)) * (np.array([61, 70]) - 1) * spacing
    out = _run((ctx, lambda o: ctx.solve2d(pos, o, precision)), dict(n_sweeps=3, tolerance=1e-6))
    _check(out, None)
    assert out[1][1] != out[0][1]
