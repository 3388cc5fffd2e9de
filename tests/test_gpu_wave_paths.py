"""Instances of the wave-step kernels that only large calls take: many models whose warp blocks
are too many to run both orderings of a pair in one launch."""
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
