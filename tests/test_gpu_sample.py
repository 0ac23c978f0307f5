"""The FP64 sample of a window taken straight from its snapshots: the bits of the packed FP64
window at the sampled groups, at the edges of blocks and strides, and the norms on top."""

import numpy as np
import pytest
import torch

from pyftle_b200 import SnapshotSeries, flows, run_window
from pyftle_b200.interpolate import GridSpec
from pyftle_b200.window import sample_error, sample_window_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("mode", ["hold", "blend"])
@pytest.mark.parametrize("integ", ["euler", "ab2", "rk4"])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("groups,stride", [(1, 100), (17, 1), (321, 20), (1000, 3)])
def test_sample_has_the_packed_windows_bits(dim, mode, integ, periodic, groups, stride):
    rng = np.random.default_rng(2)
    n = (19, 16, 17)[:dim]
    grid = GridSpec(n, (0.0,) * dim, tuple(1.0 / k for k in n), periodic)
    snaps = torch.as_tensor(rng.uniform(-1, 1, (6, dim, int(np.prod(n)))), device="cuda")
    kw = dict(precision="fx15", periodic_time=periodic, keep_source=True)
    series = SnapshotSeries(grid, snaps, **kw)
    kw.update(precision="fp64")
    cent = rng.uniform(-0.1, 1.1, (groups, dim))
    seeds = torch.as_tensor((flows.seeds_2d if dim == 2 else flows.seeds_3d)(cent, 1e-3),
                            device="cuda")
    win = dict(integrator=integ, time_mode=mode, h=0.02, num_steps=6, map_period=None, t0=0.21,
               first_snapshot=0, snapshot_t0=0.0, snapshot_dt=0.05)
    field = run_window(SnapshotSeries(grid, snaps, **kw), seeds, keep_positions=True, **win)
    out = torch.full((-(-groups // stride),), -1.0, dtype=torch.float64, device="cuda")
    sample_window_f64(series, seeds, stride, out, torch.cuda.current_stream(), **win)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), field[::stride].cpu().numpy())


@pytest.mark.parametrize("groups,stride", [(1, 1), (255, 1), (70001, 3), (400000, 1)])
def test_sample_error(groups, stride):
    rng = np.random.default_rng(3)
    f = rng.normal(size=groups)
    s = f[::stride] * (1 + 1e-3 * rng.normal(size=f[::stride].size))
    got = sample_error(torch.as_tensor(f, device="cuda"), torch.as_tensor(s, device="cuda"), stride)
    want = np.linalg.norm(f[::stride] - s) / np.linalg.norm(s)
    # sums of at most 2^19 positive terms in trees and runs: far below 1e-12
    assert got == pytest.approx(want, rel=1e-12)


def test_sample_error_of_zero_and_nan():
    z = torch.zeros(5, dtype=torch.float64, device="cuda")
    assert sample_error(z, z, 1) == 0.0
    assert sample_error(z + 2.0, z, 1) == pytest.approx(2.0 * 5 ** 0.5, rel=1e-15)
    assert np.isnan(sample_error(z * float("nan"), z, 1))
