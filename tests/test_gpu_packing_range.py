"""Snapshot packing at the ends of the value range that its header can hold."""

import numpy as np
import pytest

from pyftle_b200 import GridSpec, SnapshotSeries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("num", [1, 3, 9])
def test_fx16_ranges_whose_offset_is_past_fp32(dim, num):
    """The scale still fits FP32, the offset does not: (x + infinity) / scale is past the last
    code, NaN takes code 0; an infinite scale gives NaN for every value, code 0."""
    shape = (9, 9, 7)[:dim]
    nodes = int(np.prod(shape))
    rng = np.random.default_rng(num)
    snaps = rng.uniform(-1.0, 1.0, (num, dim, nodes))
    snaps[:, 0] = 2.5e38 * snaps[:, 0] + 1e37  # scale 3.3e38, offset -4.1e38
    snaps[0, 0, :2] = -2.4e38, 2.6e38
    snaps[:, 1] *= 3.4e38                       # scale 4.5e38
    snaps[0, 1, :2] = -3.4e38, 3.4e38
    snaps[num // 2, 0, 5] = np.nan
    grid = GridSpec(shape, (0.0,) * dim, (1.0,) * dim)
    raw = SnapshotSeries(grid, snaps, precision="fx16").packed.cpu().numpy()
    head = raw[:64].view(np.float32).reshape(4, 4)
    assert np.isfinite(head[0, 0]) and head[1, 0] == -np.inf and head[0, 1] == np.inf
    rec = raw[256:].view(np.uint16).reshape(num, nodes, 2, -1)
    nxt = np.concatenate((snaps[1:], snaps[-1:]))
    for half, x in ((0, snaps), (1, nxt)):
        np.testing.assert_array_equal(rec[:, :, half, 0], np.where(np.isnan(x[:, 0]), 0, 65535))
        assert not rec[:, :, half, 1].any()
        if dim == 3:
            assert len(np.unique(rec[:, :, half, 2])) > nodes // 2
