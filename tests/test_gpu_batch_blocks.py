"""Blocks that a batched launch puts on the GPU: as many per SM as its schedule says."""

import json
import math

import numpy as np
import pytest
import torch

from pyftle_b200 import SnapshotSeries, flows
from pyftle_b200.batch import Schedule, WindowBatch, WindowSpecRun
from pyftle_b200.interpolate import GridSpec

pytestmark = pytest.mark.gpu


def _batch(dim, sizes=(200, 300), **kw):
    n = 16
    grid = GridSpec((n,) * dim, (0.0,) * dim, (2 * math.pi / n,) * dim, True)
    rng = np.random.default_rng(dim)
    series = SnapshotSeries(grid, rng.uniform(-1, 1, (5, dim, n ** dim)), precision="fx15")
    seeds = flows.seeds_2d if dim == 2 else flows.seeds_3d
    runs = [WindowSpecRun(torch.as_tensor(seeds(rng.uniform(0, 2 * math.pi, (m, dim)), 1e-3),
                                          device="cuda"), 0.0, 0.01, 4, keep_positions=True)
            for m in sizes]
    return WindowBatch(series, runs, snapshot_dt=0.1, **kw)


def _grid(run, tmp_path):
    """Blocks of the batched kernel's launch, from the profiler's record of it."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU,
                                            torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        events = json.load(f)["traceEvents"]
    if not any(e.get("cat") == "kernel" for e in events):
        pytest.skip("the profiler records no kernels on this machine")
    grids = [e["args"]["grid"] for e in events if "windows_persistent_kernel" in e.get("name", "")
             and "grid" in e.get("args", {})]
    assert len(grids) == 1
    return math.prod(grids[0])


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("blocks", [1, 3, 4, 8])
def test_a_schedule_is_the_blocks_per_sm(dim, blocks, tmp_path):
    batch = _batch(dim)
    batch.run()
    assert _grid(lambda: batch.run(Schedule(blocks, 1)), tmp_path) == 148 * blocks


@pytest.mark.parametrize("dim", [2, 3])
def test_few_work_items_run_on_4_blocks_per_sm(dim, tmp_path):
    batch = _batch(dim)
    batch.run()
    assert _grid(batch.run, tmp_path) == 148 * 4


@pytest.mark.parametrize("precision", ["fx15", "fx16", "fp16", "bf16"])
@pytest.mark.parametrize("peak,blocks", [(0.5, 8), (1e5, 4)])
def test_many_work_items_run_on_8_blocks_where_groups_stay_compact(precision, peak, blocks,
                                                                   tmp_path):
    peak = min(peak, 6e4) if precision == "fp16" else peak
    n, groups = 16, 9 * 148 * 128
    grid = GridSpec((n, n), (0.0, 0.0), (2 * math.pi / n,) * 2, True)
    rng = np.random.default_rng(8)
    snaps = rng.uniform(-0.25, 0.25, (3, 2, n * n)) * peak
    snaps[1, 1, 7] = -peak
    series = SnapshotSeries(grid, snaps, precision=precision)
    assert series.peak_speed() == pytest.approx(peak, rel=2.0 ** -8)
    seeds = torch.as_tensor(flows.seeds_2d(rng.uniform(0, 6, (groups, 2)), 1e-3), device="cuda")
    batch = WindowBatch(series, [WindowSpecRun(seeds, 0.0, 0.01, 4, keep_positions=True)],
                        snapshot_dt=0.1)
    assert batch.schedule == Schedule(blocks, 1)
    batch.run()
    assert _grid(batch.run, tmp_path) == 148 * blocks
