"""Cell location of the FP64 window kernels against the CPU oracle, where it can go wrong.

The kernels divide by the spacing through its reciprocal, take floors by a rounding
addition, wrap periodic cells without a modulo where they can, share time lookups within a
warp and reuse a stage's corner values: every one of these has to leave the oracle's bits.
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyftle_b200 import GridSpec, SnapshotSeries, run_window

pytestmark = pytest.mark.gpu

# spacings next to powers of two (mantissas of all ones and of one bit), ordinary, extreme
SPACINGS = [0.5, np.nextafter(0.5, 0), np.nextafter(0.5, 1), 1.0 / 3.0, 2 * np.pi / 7, 1e-3,
            2.0 ** -310 * 1.3, 2.0 ** 305 * 1.7]


def _case(dim, periodic, spacing, seed, n_groups):
    rng = np.random.default_rng(seed)
    shape = (7, 7, 5)[:dim]
    origin = tuple((-3.0 * spacing, 0.0, 0.25 * spacing)[:dim])
    grid = GridSpec(shape, origin, (spacing,) * dim, periodic)
    nodes = int(np.prod(shape))
    snaps = rng.standard_normal((6, dim, nodes)) * spacing
    snaps[:, :, rng.integers(0, nodes, 3)] = 0.0
    span = np.array(shape) * spacing
    pos = np.array(origin) + span * rng.uniform(-0.1, 1.1, (2 * dim * n_groups, dim))
    # points on nodes and faces, at the origin, next to it, far away and not finite
    k = min(len(pos), 40)
    odd = pos[rng.permutation(len(pos))[:k]]
    odd[0::5] = origin
    odd[1::5] = np.array(origin) + spacing * rng.integers(0, 7, odd[1::5].shape)
    odd[2::5] = np.nextafter(np.array(origin), 1e300 * (-1) ** np.arange(dim))
    odd[3::5] += 37.0 * span if periodic else span
    odd[4::5, 0] = [np.nan, np.inf, -np.inf, -0.0, 0.0, 1e-290, -1e-290, 5e-324][:odd[4::5].shape[0]]
    pos[rng.permutation(len(pos))[:k]] = odd
    return grid, snaps, pos


@pytest.mark.parametrize("spacing", SPACINGS)
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_window_positions_keep_the_oracles_bits(dim, periodic, spacing):
    # HOLD and BLEND, group counts around a warp's and a block's, steps around the shared
    # time lookups' 10 (RK4) and 32 (Euler, AB2), forward and backward
    for i, (mode, integrator, steps, n_groups, h) in enumerate([
            ("hold", "rk4", 6, 33, 0.3), ("hold", "ab2", 5, 16, -0.3), ("blend", "rk4", 10, 1, 0.3),
            ("blend", "rk4", 21, 129, 0.25), ("blend", "rk4", 9, 31, -0.4),
            ("blend", "euler", 33, 17, 0.1), ("blend", "ab2", 32, 64, 0.1)]):
        grid, snaps, pos = _case(dim, periodic, spacing, 100 + i, n_groups)
        kw = dict(integrator=integrator, h=h, num_steps=steps)
        if mode == "blend":
            kw.update(t0=0.05, snap_dt=0.7)
        p_ref, f_ref = O.run_window(snaps, grid.shape, grid.origin, grid.spacing, pos,
                                    time_mode=O.HOLD if mode == "hold" else O.BLEND,
                                    periodic_space=periodic, periodic_time=mode == "blend", **kw)
        series = SnapshotSeries(grid, snaps, periodic_time=mode == "blend")
        p = torch.as_tensor(pos, device="cuda")
        if mode == "blend":
            kw["snapshot_dt"] = kw.pop("snap_dt")
        f = run_window(series, p, time_mode=mode, **kw)
        np.testing.assert_array_equal(p.cpu().numpy(), p_ref)
        np.testing.assert_allclose(f.cpu().numpy(), f_ref, rtol=1e-12, atol=1e-13)
