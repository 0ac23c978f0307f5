"""Grid spacings at the end of what a grid accepts: (x - origin) / spacing as IEEE division
gives it, so an infinite spacing leaves a point on the grid's first plane."""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyftle_b200 import GridSpec, SnapshotSeries, run_window
from pyftle_b200.interpolate import create_interpolator

pytestmark = pytest.mark.gpu

X = [0.25, 0.5, -0.75, 1e-300, 5e-324, 0.0, -0.0, 1e300, -1e300, 1.7e308, np.inf, -np.inf, np.nan]


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_infinite_spacing(periodic, axis, sign):
    shape, spacing = (6, 5), [0.5, 0.5]
    spacing[axis] = sign * np.inf
    grid = GridSpec(shape, (-1.0, -1.0), tuple(spacing), periodic)
    snaps = np.random.default_rng(4).standard_normal((4, 2, 30))
    pts = np.array([(a, b) for a in X for b in X])[:4 * (len(X) ** 2 // 4)]
    interp = create_interpolator("grid", shape, periodic=periodic)
    interp.grid, interp.snapshot = grid, torch.as_tensor(snaps[0], device="cuda")
    with np.errstate(all="ignore"):
        p = (pts + 1.0) / np.array(spacing)  # the index coordinates
        fl = np.floor(p)
        ok = (np.abs(fl) < 1e9).all(1) if periodic else ((p >= 0) & (p < np.array(shape) - 1)).all(1)
    i = np.where(ok[:, None], fl, 0).astype(int)
    f = np.where(ok[:, None], p - i, 0.0)
    j = [i % np.array(shape), (i + 1) % np.array(shape)]
    v = lambda a, b: snaps[0][:, j[b][:, 1] * 6 + j[a][:, 0]].T  # noqa: E731
    x, y = f[:, :1], f[:, 1:]
    want = (v(0, 0) * (1 - x) * (1 - y) + v(1, 0) * x * (1 - y) + v(0, 1) * (1 - x) * y
            + v(1, 1) * x * y)
    want[~ok] = 0.0
    assert ok.any()
    got = interp.interpolate(torch.as_tensor(pts, device="cuda")).cpu().numpy()
    np.testing.assert_array_equal(got, want)
    # the windows locate a point in the same way
    pos = torch.as_tensor(pts, device="cuda")
    run_window(SnapshotSeries(grid, snaps), pos, time_mode="hold", integrator="euler", h=0.1,
               num_steps=4, with_ftle=False)
    want, _ = O.run_window(snaps, shape, grid.origin, grid.spacing, pts, integrator="euler",
                           time_mode=O.HOLD, periodic_space=periodic, h=0.1, num_steps=4)
    np.testing.assert_array_equal(pos.cpu().numpy(), want)
