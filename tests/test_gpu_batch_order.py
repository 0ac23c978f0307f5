"""Batched windows whose groups are taken in spatial order: the caller's buffers hold the
bits that the given order leaves there, whichever way the order reaches the kernel."""

import math

import numpy as np
import pytest
import torch

from pyftle_b200 import SnapshotSeries, flows
from pyftle_b200.batch import Schedule, WindowBatch, WindowSpecRun
from pyftle_b200.interpolate import GridSpec

pytestmark = pytest.mark.gpu


def _series(dim):
    n = 24
    grid = GridSpec((n,) * dim, (0.0,) * dim, (2 * math.pi / n,) * dim, True)
    return SnapshotSeries(grid, np.random.default_rng(1).uniform(-1, 1, (6, dim, n ** dim)),
                          precision="fx15")


def _run(series, dim, order, sizes, keep, share, exchange):
    rng = np.random.default_rng(7)
    seeds = flows.seeds_2d if dim == 2 else flows.seeds_3d
    bufs = [torch.as_tensor(seeds(rng.uniform(0, 2 * math.pi, (n, dim)), 1e-3), device="cuda")
            for n in sizes]
    if share:  # the windows read and write one buffer
        bufs = [bufs[-1]] * len(bufs)
    runs = [WindowSpecRun(b, 0.1 * i, 0.01, 9 + i, keep_positions=keep)
            for i, b in enumerate(bufs)]
    if share == "ftle":
        for w in runs[1:]:
            w.ftle = runs[0].ftle = torch.empty(sizes[-1], dtype=torch.float64, device="cuda")
    batch = WindowBatch(series, runs, snapshot_dt=0.1, spatial_order=order)
    if exchange:
        batch.run(Schedule(4, 1))
        for w in runs:
            w.ftle = torch.full_like(w.ftle, -1.0)
    out = batch.run(Schedule(4, 1))
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out], [b.cpu().numpy() for b in bufs], batch


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("sizes", [(1,), (127, 128, 129), (3, 700)])
def test_spatial_order_leaves_the_same_bits(dim, keep, sizes):
    a = _run(_series(dim), dim, False, sizes, keep, False, False)
    b = _run(_series(dim), dim, True, sizes, keep, False, False)
    for x, y in zip(a[0] + a[1], b[0] + b[1]):
        np.testing.assert_array_equal(x, y)


def test_exchanged_ftle_buffers_receive_the_result():
    sizes = (127, 300)
    a = _run(_series(2), 2, True, sizes, True, False, False)
    b = _run(_series(2), 2, True, sizes, True, False, True)
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)


def test_read_only_seeds_with_a_shared_ftle_buffer_keep_the_last_window():
    sizes = (300, 300)
    alone = _run(_series(2), 2, True, sizes, True, True, False)
    shared = _run(_series(2), 2, True, sizes, True, "ftle", False)
    np.testing.assert_array_equal(shared[0][1], alone[0][1])
