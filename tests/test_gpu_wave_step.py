"""The wave-step 3D kernel (the default on uniform grids) at the edges of its 8 x 4 warp block, of
its 4-node ring chunks and of its group of four steps, against the oracle, bit for bit."""
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
@pytest.mark.parametrize("grid", GRIDS)
def test_wave_step_block_edges_match_the_oracle(ctx, oracle, grid, precision, near):
    nx, ny, nz = grid
    h = 50.0
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    dt = np.float32 if precision == ex.F32 else np.float64
    s = random_slowness(rng, (nz - 1) * (ny - 1) * (nx - 1), dtype=dt)
    ctx.set_grid3d(nx, ny, nz, h, h, h)
    ctx.set_slowness3d(s)
    ends = np.array([(nx - 1) * h, (ny - 1) * h, (nz - 1) * h])
    pos = np.concatenate([[[0.0, 0.0, 0.0], ends], rng.uniform(0, 1, (4, 3)) * ends])
    opt = ex.Options(n_sweeps=3, tolerance=1e-6, factored_radius=2, near_fp64=near)
    t = ctx.solve3d(pos, opt, precision)
    for p, a in zip(pos, t):
        cell = [min(n - 2, int(q / h)) for q, n in zip(p, grid)]
        ref = oracle.solve3d(s, (nx, ny, nz, h, h, h), cell, p, n_sweeps=3, radius=2, tol=1e-6, near_fp64=near)
        assert np.array_equal(_bits(a), _bits(ref)), (p, np.abs(a - ref).max())
