"""What eikx_autotune3d reports names the kernel that it chose, and tables written before the
default kernel was a candidate no longer decide.  The kernels of a solve show in its launches: the
default runs both orderings of a pair in one, the others do not."""
import json

import numpy as np
import pytest

from conftest import random_slowness

pytestmark = pytest.mark.gpu

import eikonalxx_gb300 as ex  # noqa: E402

GRID = (45, 38, 27, 50.0, 50.0, 50.0)
SRC = [(300.0, 700.0, 200.0), (1500.0, 100.0, 900.0)]


def _context(rng):
    c = ex.Context(0)
    c.set_grid3d(*GRID)
    c.set_slowness3d(random_slowness(rng, (GRID[0] - 1) * (GRID[1] - 1) * (GRID[2] - 1), dtype=np.float32))
    return c


def _launches(c, **opt):
    c.solve3d(SRC, ex.Options(n_sweeps=3, tolerance=-1, **opt), ex.F32)
    return c.stats()["kernel_launches"]


def test_the_reported_choice_can_be_asked_for():
    with _context(np.random.default_rng(6)) as c:
        wave, chunk = _launches(c), _launches(c, sweep_kernel=2)
        assert wave != chunk
        t = c.autotune3d(SRC, ex.F32)
        if t["wave_step"]:
            asked = dict(blocks_per_sm=t["blocks_per_sm"])
        else:
            asked = {k: t[k] for k in ("sweep_kernel", "pair_fields", "block_shape", "blocks_per_sm")}
        assert _launches(c, **asked) == _launches(c) == (wave if t["wave_step"] else chunk)


def test_tables_without_the_default_kernel_are_left_out(tmp_path):
    rng = np.random.default_rng(6)
    entry = {"precision": ex.F32, "uniform": 1, "nx": 64, "ny": 64, "nz": 32, "nsrc": 2, "sweep_kernel": 2, "pair_fields": 0,
             "block_shape": 1, "blocks_per_sm": 4, "ms_per_sweep": 0.1, "default_ms_per_sweep": 0.1, "candidates": 8}
    path = tmp_path / "tuning.jsonl"
    for mark in ({}, {"wave": 0}, {"wave": 1}):
        path.write_text(json.dumps({**entry, **mark}) + "\n")
        with _context(rng) as c:
            wave, chunk = _launches(c), _launches(c, sweep_kernel=2)
            c.load_tuning(str(path))
            assert _launches(c) == (chunk if mark == {"wave": 0} else wave)
            c.save_tuning(str(tmp_path / "again.jsonl"))
        rows = [json.loads(line) for line in (tmp_path / "again.jsonl").read_text().splitlines()]
        assert [r["wave"] for r in rows] == list(mark.values())
