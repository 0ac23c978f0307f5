"""16-bit windows: a group's result does not depend on the groups beside it, also where those
take the rare branches of the advection kernel (seeds that are not finite, outside the grid or
many periods away)."""

import numpy as np
import pytest
import torch

from pyftle_b200 import SnapshotSeries, flows, run_window
from pyftle_b200.interpolate import GridSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("chunk", [None, 3])
def test_odd_neighbours_leave_a_group_alone(dim, periodic, chunk):
    rng = np.random.default_rng(11)
    n = (19, 16, 17)[:dim]
    grid = GridSpec(n, (0.0,) * dim, tuple(1.0 / k for k in n), periodic)
    series = SnapshotSeries(grid, rng.uniform(-1, 1, (4, dim, int(np.prod(n)))),
                            precision="fx15")
    cent = rng.uniform(0.2, 0.7, (257, dim))
    odd = rng.integers(0, 2, 257).astype(bool)
    cent_odd = cent.copy()
    cent_odd[odd] = np.resize([np.nan, np.inf, -40.3, 7.2, 1e11, 0.9999], (odd.sum(), 1))
    out = []
    for c in (cent, cent_odd):
        seeds = (flows.seeds_2d if dim == 2 else flows.seeds_3d)(c, 2e-2)
        pos = torch.as_tensor(seeds, device="cuda")
        f = run_window(series, pos, integrator="rk4", time_mode="blend", h=0.02, num_steps=7,
                       snapshot_dt=0.06, chunk_steps=chunk)
        torch.cuda.synchronize()
        out.append((f.cpu().numpy()[~odd], pos.view(2 * dim, -1, dim).cpu().numpy()[:, ~odd]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert np.isfinite(out[0][0]).all()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("integ", ["euler", "ab2", "rk4"])
@pytest.mark.parametrize("groups", [1, 127, 129, 4000])
@pytest.mark.parametrize("sort_every", [0, 1, 2])
def test_chunks_keep_the_bits_of_one_launch(dim, integ, groups, sort_every):
    """Groups travel from chunk to chunk through the sort's order: records, tags and AB2
    history arrive with their group, whichever chunks are sorted."""
    rng = np.random.default_rng(4)
    n = (19, 16, 17)[:dim]
    grid = GridSpec(n, (0.0,) * dim, tuple(1.0 / k for k in n), True)
    series = SnapshotSeries(grid, rng.uniform(-3, 3, (4, dim, int(np.prod(n)))),
                            precision="fx15")
    seeds = (flows.seeds_2d if dim == 2 else flows.seeds_3d)(
        rng.uniform(0, 1, (groups, dim)), 5e-3)
    out = []
    for chunk in (None, 3):
        pos = torch.as_tensor(seeds, device="cuda")
        f = run_window(series, pos, integrator=integ, time_mode="blend", h=0.02, num_steps=14,
                       snapshot_dt=0.1, chunk_steps=chunk, sort_every=sort_every)
        torch.cuda.synchronize()
        out.append((f.cpu().numpy(), pos.cpu().numpy()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
