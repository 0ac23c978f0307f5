"""A batch run on a stream of its own after its buffers were exchanged: the results reach the
new buffers, and the old ones live as long as the plan that points at them."""

import gc
import math
import weakref

import numpy as np
import pytest
import torch

from pyftle_b200 import SnapshotSeries, flows
from pyftle_b200.batch import WindowBatch, WindowSpecRun
from pyftle_b200.interpolate import GridSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keep", [False, True])
def test_exchange_then_run_on_a_side_stream(keep):
    n, groups = 24, 300
    grid = GridSpec((n, n), (0.0, 0.0), (2 * math.pi / n,) * 2, True)
    rng = np.random.default_rng(3)
    series = SnapshotSeries(grid, rng.uniform(-1, 1, (6, 2, n * n)), precision="fx15")
    seeds = torch.as_tensor(flows.seeds_2d(rng.uniform(0, 2 * math.pi, (groups, 2)), 1e-3),
                            device="cuda")

    def batch(positions):
        w = WindowSpecRun(positions, 0.1, 0.01, 12, keep_positions=keep)
        return w, WindowBatch(series, [w], snapshot_dt=0.1)

    want_window, want = batch(seeds.clone())
    want.run()
    window, b = batch(seeds.clone())
    b.run()
    old = weakref.ref(window.ftle)
    if not keep:
        window.positions.copy_(seeds)  # the next run reads the batch's own seed buffer
    window.positions, window.ftle = torch.zeros_like(seeds), torch.full_like(window.ftle, -1.0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    b.run(stream=side)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    gc.collect()
    assert old() is not None  # the first plan still holds its address
    assert torch.equal(window.ftle, want_window.ftle)
    if not keep:
        assert torch.equal(window.positions, want_window.positions)
    blocks = {s["stream"] for s in torch.cuda.memory_snapshot()
              for t in b._sorted + [f for _, f in b._bound]
              if s["address"] <= t.data_ptr() < s["address"] + s["total_size"]}
    assert blocks == {side.cuda_stream}
