"""Routes of a 3D solve that few calls take: many models whose warp blocks are too many to run both
orderings of a pair in one launch, and one source on a long thin non-uniform grid."""
import numpy as np
import pytest

from conftest import random_slowness

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import eikonalxx_gb300 as ex  # noqa: E402


def _bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


# fields of 5 x 8 warp blocks, four resident warps per SM: above ten blocks a warp the orderings run
# one by one, and on the warps of all resident blocks (two per SM at least) both share a launch
@pytest.mark.parametrize("precision,near", [(ex.F32, False), (ex.F32, True), (ex.F64, False)])
@pytest.mark.parametrize("spacing", [(50.0, 50.0, 50.0), (50.0, 65.0, 40.0)])
def test_many_models_one_ordering_per_launch(ctx, oracle, spacing, precision, near):
    grid = nx, ny, nz = 41, 34, 30
    fields = torch.cuda.get_device_properties(0).multi_processor_count + 8
    rng = np.random.default_rng(17)
    dt = np.float32 if precision == ex.F32 else np.float64
    models = []
    for k in range(4):
        n = fields // 4 + (1 if k < fields % 4 else 0)
        models.append({"grid": grid + spacing, "model": random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=dt),
                       "sources": rng.uniform(0, 1, (n, 3)) * (np.array(grid) - 1) * spacing})
    opt = dict(n_sweeps=4, tolerance=1e-5, near_fp64=near)
    runs = []
    for per_sm in (0, 1):
        t = ctx.solve3d_batch(models, ex.Options(**opt, blocks_per_sm=per_sm), precision)
        runs.append((t, ctx.stats()))
    # both orderings: two launches fewer than one by one in the initialisation, at least
    assert runs[0][1]["kernel_launches"] != runs[1][1]["kernel_launches"]
    for k in ("iterations_max", "iterations_min", "sweeps_launched", "refine_node_updates"):
        assert runs[0][1][k] == runs[1][1][k]
    for a, b in zip(runs[0][0], runs[1][0]):
        assert np.array_equal(_bits(a), _bits(b))
    for m, out in zip(models, runs[1][0]):
        p = m["sources"][-1]
        cell = [min(n - 2, int(q / h)) for q, n, h in zip(p, grid, spacing)]
        ref = oracle.solve3d(m["model"], (nx, ny, nz, *spacing), cell, p, n_sweeps=4, radius=3, tol=1e-5, near_fp64=near)
        assert np.array_equal(_bits(out[-1]), _bits(ref))


# at the line nx = 3 (ny + nz)^2, and past 60 (ny + nz) below it; one source, non-uniform: chunk-step
@pytest.mark.parametrize("precision,near", [(ex.F32, False), (ex.F32, True), (ex.F64, False)])
@pytest.mark.parametrize("grid,spacing,sources,chunk", [((108, 3, 3), (50.0, 65.0, 40.0), 1, True), ((107, 3, 3), (50.0, 65.0, 40.0), 1, False),
                                                        ((1321, 15, 7), (50.0, 65.0, 40.0), 1, True), ((108, 3, 3), (50.0, 65.0, 40.0), 2, False),
                                                        ((108, 3, 3), (50.0, 50.0, 50.0), 1, False)])
def test_one_source_on_a_long_thin_grid(ctx, oracle, grid, spacing, sources, chunk, precision, near):
    nx, ny, nz = grid
    rng = np.random.default_rng(19)
    dt = np.float32 if precision == ex.F32 else np.float64
    s = random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=dt)
    ctx.set_grid3d(*grid, *spacing)
    ctx.set_slowness3d(s)
    pos = rng.uniform(0, 1, (sources, 3)) * (np.array(grid) - 1) * spacing
    opt = dict(n_sweeps=2, tolerance=-1, near_fp64=near)
    ctx.solve3d(pos, ex.Options(**opt, sweep_kernel=2), precision)
    launches = ctx.stats()["kernel_launches"]
    t = ctx.solve3d(pos, ex.Options(**opt), precision)
    assert (ctx.stats()["kernel_launches"] == launches) == chunk
    for p, a in zip(pos, t):
        cell = [min(n - 2, int(q / h)) for q, n, h in zip(p, grid, spacing)]
        ref = oracle.solve3d(s, (nx, ny, nz, *spacing), cell, p, n_sweeps=2, radius=3, near_fp64=near)
        assert np.array_equal(_bits(a), _bits(ref))
