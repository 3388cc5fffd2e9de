"""The wave-step kernels (the 3D and 2D defaults) at the edges of their
warp blocks (8 x 4 rows, 32 rows), of their 4-node ring chunks and of their groups of four steps,
against the oracle, bit for bit."""
import numpy as np
import pytest

from conftest import random_slowness

pytestmark = pytest.mark.gpu

import eikonalxx_gb300 as ex  # noqa: E402


def _bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


# extents: a warp block's rows start at the first updated row (index 1), so ny - 1 = 7, 8, 9, 17
# and nz - 1 = 3, 4, 5, 9 straddle the block; nx = 3 .. 6, 31 .. 34 the chunk and the walk's ends
GRIDS = [(3, 8, 4), (4, 9, 5), (5, 10, 6), (6, 18, 10), (31, 9, 10), (32, 10, 5), (33, 17, 6), (34, 18, 4)]


@pytest.mark.parametrize("precision,near", [(ex.F32, False), (ex.F32, True), (ex.F64, False)])
@pytest.mark.parametrize("spacing", [(50.0, 50.0, 50.0), (50.0, 65.0, 8.0)])
@pytest.mark.parametrize("grid", GRIDS)
def test_wave_step_block_edges_match_the_oracle(ctx, oracle, grid, spacing, precision, near):
    nx, ny, nz = grid
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    dt = np.float32 if precision == ex.F32 else np.float64
    s = random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=dt)
    ctx.set_grid3d(nx, ny, nz, *spacing)
    ctx.set_slowness3d(s)
    ends = (np.array(grid) - 1) * spacing
    pos = np.concatenate([[[0.0, 0.0, 0.0], ends], rng.uniform(0, 1, (4, 3)) * ends])
    opt = ex.Options(n_sweeps=3, tolerance=1e-6, factored_radius=2, near_fp64=near)
    t = ctx.solve3d(pos, opt, precision)
    for p, a in zip(pos, t):
        cell = [min(n - 2, int(q / h)) for q, n, h in zip(p, grid, spacing)]
        ref = oracle.solve3d(s, (nx, ny, nz, *spacing), cell, p, n_sweeps=3, radius=2, tol=1e-6, near_fp64=near)
        assert np.array_equal(_bits(a), _bits(ref)), (p, np.abs(a - ref).max())


# rows from the first updated one: nz - 1 = 31, 32, 33, 65 straddle the 32-row block; h = 0.01
# (kilometres) makes the cell-edge operators t1 + h sqrt(.) the smallest ones, h = 10 the others
GRIDS2 = [(3, 32), (4, 33), (5, 34), (6, 66), (33, 33), (34, 34), (61, 40)]


@pytest.mark.parametrize("precision", [ex.F32, ex.F64])
@pytest.mark.parametrize("spacing", [(10.0, 10.0), (0.01, 0.01), (10.0, 12.5)])
@pytest.mark.parametrize("grid", GRIDS2)
def test_wave_step_2d_block_edges_match_the_oracle(ctx, oracle, grid, spacing, precision):
    nx, nz = grid
    dx, dz = spacing
    rng = np.random.default_rng(nx * 100 + nz)
    dt = np.float32 if precision == ex.F32 else np.float64
    s = random_slowness(rng, (nz - 1) * (nx - 1), dtype=dt)
    if dx < 1:
        s = (s * 1000).astype(dt)
    ctx.set_grid2d(nx, nz, dx, dz)
    ctx.set_slowness2d(s)
    ends = np.array([(nx - 1) * dx, (nz - 1) * dz])
    pos = np.concatenate([[[0.0, 0.0], ends], rng.uniform(0, 1, (3, 2)) * ends])
    t = ctx.solve2d(pos, ex.Options(n_sweeps=3, tolerance=1e-9, factored_radius=2), precision)
    for p, a in zip(pos, t):
        cell = [min(n - 2, int(q / d)) for q, n, d in zip(p, grid, spacing)]
        ref = oracle.solve2d(s, (nx, nz, dx, dz), cell, p, n_sweeps=3, radius=2, tol=1e-9)
        assert np.array_equal(_bits(a), _bits(ref)), (p, np.abs(a - ref).max())


# 160 fields of 5 x 8 warp blocks: on the warps of four (two in double) resident blocks per SM both
# orderings of a pair share a launch, on those of one they don't
@pytest.mark.parametrize("precision", [ex.F32, ex.F64])
@pytest.mark.parametrize("spacing", [(50.0, 50.0, 50.0), (50.0, 65.0, 40.0)])
@pytest.mark.parametrize("init,tol", [(True, 1e-2), (True, 1e-4), (True, 1e-5), (True, 1e-6), (False, 1e-4)])
def test_both_orderings_in_one_launch_match_one_by_one(ctx, oracle, spacing, precision, init, tol):
    grid = nx, ny, nz = 41, 34, 30
    rng = np.random.default_rng(11)
    dt = np.float32 if precision == ex.F32 else np.float64
    s = random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=dt)
    ctx.set_grid3d(nx, ny, nz, *spacing)
    ctx.set_slowness3d(s)
    pos = rng.uniform(0, 1, (160, 3)) * (np.array(grid) - 1) * spacing
    out = []
    for per_sm in (0, 1):
        t = ctx.solve3d(pos, ex.Options(n_sweeps=6, tolerance=tol, init_sweeps=init, blocks_per_sm=per_sm), precision)
        st = ctx.stats()
        out.append((t, [st[k] for k in ("iterations_max", "iterations_min", "sweeps_launched", "refine_node_updates")]))
    assert out[0][1] == out[1][1]
    assert np.array_equal(_bits(np.asarray(out[0][0])), _bits(np.asarray(out[1][0])))
    for i in (0, 77, 159):
        cell = [min(n - 2, int(q / h)) for q, n, h in zip(pos[i], grid, spacing)]
        ref = oracle.solve3d(s, (nx, ny, nz, *spacing), cell, pos[i], n_sweeps=6, radius=3, tol=tol, init_sweeps=init)
        assert np.array_equal(_bits(out[0][0][i]), _bits(ref))


# 2100 fields of 3 warp blocks, likewise
@pytest.mark.parametrize("precision", [ex.F32, ex.F64])
@pytest.mark.parametrize("spacing", [(10.0, 10.0), (10.0, 12.5)])
@pytest.mark.parametrize("init,tol", [(True, 1e-3), (True, 1e-5), (True, 1e-7), (False, 1e-5)])
def test_both_orderings_in_one_launch_match_one_by_one_2d(ctx, oracle, spacing, precision, init, tol):
    grid = nx, nz = 23, 66
    rng = np.random.default_rng(12)
    dt = np.float32 if precision == ex.F32 else np.float64
    s = random_slowness(rng, (nz - 1) * (nx - 1), dtype=dt)
    ctx.set_grid2d(nx, nz, *spacing)
    ctx.set_slowness2d(s)
    pos = rng.uniform(0, 1, (2100, 2)) * (np.array(grid) - 1) * spacing
    out = []
    for per_sm in (0, 1):
        t = ctx.solve2d(pos, ex.Options(n_sweeps=6, tolerance=tol, init_sweeps=init, blocks_per_sm=per_sm), precision)
        st = ctx.stats()
        out.append((t, [st[k] for k in ("iterations_max", "iterations_min", "sweeps_launched", "refine_node_updates")]))
    assert out[0][1] == out[1][1]
    assert np.array_equal(_bits(np.asarray(out[0][0])), _bits(np.asarray(out[1][0])))
    for i in (0, 1033, 2099):
        cell = [min(n - 2, int(q / h)) for q, n, h in zip(pos[i], grid, spacing)]
        ref = oracle.solve2d(s, (nx, nz, *spacing), cell, pos[i], n_sweeps=6, radius=3, tol=tol, init_sweeps=init)
        assert np.array_equal(_bits(out[0][0][i]), _bits(ref))
