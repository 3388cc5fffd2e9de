"""Warm starts from initial times that no solve produces: below zero, not a number, infinite or
huge.  Where the gate keeps them (a large gate_tol), the default kernel's times are those of the
kernels that evaluate every operator, bit for bit."""
import numpy as np
import pytest

from conftest import random_slowness

pytestmark = pytest.mark.gpu

import eikonalxx_gb300 as ex  # noqa: E402


def _bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


def _start(cold, kind, rng):
    """The second field's start: the cold one with a patch, or a few nodes, of other values."""
    t = cold.copy()
    f = t[1]
    patch = (slice(3, 9), slice(5, 14), slice(6, 17))
    if kind == "negative patch":
        f[patch] = rng.uniform(-2.0, -0.1, f[patch].shape)
    elif kind == "all negative":
        f[...] -= 100.0
    elif kind == "nan patch":
        f[patch] = np.nan
    elif kind == "minus nan patch":
        f[patch] = np.copysign(np.nan, -1.0)
    elif kind == "infinite patch":
        f[patch] = np.inf
    elif kind == "huge patch":
        f[patch] = 1e35
    else:   # isolated nodes just below zero
        f[2::5, 2::5, 2::5] = -1e-3
    return t


KINDS = ["negative patch", "all negative", "nan patch", "minus nan patch", "infinite patch", "huge patch", "negative nodes"]


@pytest.mark.parametrize("precision", [ex.F32, ex.F64])
@pytest.mark.parametrize("spacing", [(50.0, 50.0, 50.0), (50.0, 65.0, 40.0)])
@pytest.mark.parametrize("kind", KINDS)
def test_any_start_gives_the_operators_times(ctx, kind, spacing, precision):
    nx, ny, nz = 37, 26, 18
    rng = np.random.default_rng(81)
    s = random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=np.float32)
    ctx.set_grid3d(nx, ny, nz, *spacing)
    ctx.set_slowness3d(s)
    pos = rng.uniform(0, 1, (2, 3)) * (np.array([nx, ny, nz]) - 1) * spacing
    cold = ctx.solve3d(pos, ex.Options(n_sweeps=3, tolerance=-1), precision)
    init = _start(cold, kind, rng)
    opt = dict(n_sweeps=2, tolerance=-1, factored_radius=2)
    t = ctx.solve3d_warm(pos, init, ex.Options(**opt), precision, gate_tol=1e9)
    ref = ctx.solve3d_warm(pos, init, ex.Options(**opt, sweep_kernel=1), precision, gate_tol=1e9)
    assert np.array_equal(_bits(t), _bits(ref)), np.count_nonzero(_bits(t) != _bits(ref))


# the FP64 factor has no node-step form; the chunk-step kernel's bounds hold for infinite and huge
# times, and for times below zero beside larger positive ones
@pytest.mark.parametrize("spacing", [(50.0, 50.0, 50.0), (50.0, 65.0, 40.0)])
@pytest.mark.parametrize("kind", ["infinite patch", "huge patch", "negative nodes"])
def test_any_start_with_the_fp64_factor(ctx, kind, spacing):
    nx, ny, nz = 37, 26, 18
    rng = np.random.default_rng(82)
    s = random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=np.float32)
    ctx.set_grid3d(nx, ny, nz, *spacing)
    ctx.set_slowness3d(s)
    pos = rng.uniform(0, 1, (2, 3)) * (np.array([nx, ny, nz]) - 1) * spacing
    cold = ctx.solve3d(pos, ex.Options(n_sweeps=3, tolerance=-1, near_fp64=True), ex.F32)
    init = _start(cold, kind, rng)
    opt = dict(n_sweeps=2, tolerance=-1, factored_radius=2, near_fp64=True)
    t = ctx.solve3d_warm(pos, init, ex.Options(**opt), ex.F32, gate_tol=1e9)
    ref = ctx.solve3d_warm(pos, init, ex.Options(**opt, sweep_kernel=2), ex.F32, gate_tol=1e9)
    assert np.array_equal(_bits(t), _bits(ref)), np.count_nonzero(_bits(t) != _bits(ref))
