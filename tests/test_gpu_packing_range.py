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


# The range pass walks (snapshot, piece of 2048 nodes) with 1,184 blocks a component: more pieces
# than that over many snapshots, and in one plane, with the extremes in the last ones.
@pytest.mark.parametrize("shape,num", [((61, 41), 1400), ((1600, 1523), 2), ((1600, 1523), 5),
                                       ((17, 17, 9), 1301)])
@pytest.mark.parametrize("precision", ["fx15", "fx16"])
def test_ranges_over_more_pieces_than_blocks(precision, shape, num):
    dim, nodes = len(shape), int(np.prod(shape))
    assert num * -(-nodes // 2048) > 1184
    rng = np.random.default_rng(num)
    snaps = rng.uniform(-1.0, 1.0, (num, dim, nodes))
    snaps[-1, 0, nodes - 1], snaps[-1, 0, nodes - 1500] = 7.5, -3.25
    snaps[-1, 1, nodes // 2], snaps[0, 1, nodes - 3] = 4.5, -2.5
    raw = SnapshotSeries(GridSpec(shape, (0.0,) * dim, (1.0,) * dim), snaps,
                         precision=precision).packed.cpu().numpy()
    head = raw[:64].view(np.float32).reshape(4, 4).astype(np.float64)
    np.testing.assert_array_equal(head[2, :2], [-3.25, -2.5])
    np.testing.assert_array_equal(head[3, :2], [7.5, 4.5])
    half = 2 if dim == 2 else 4
    rec = raw[256:].view(np.uint16).reshape(num, nodes, 2, half)
    nxt = np.concatenate((snaps[1:], snaps[-1:]))
    for c in range(dim):
        for j, series in enumerate((snaps, nxt)):
            x = series[:, c]
            if precision == "fx15":
                q = np.rint((x - head[2, c]) * (32767 / (head[3, c] - head[2, c])))
                q = np.clip(q, 0, 32767)
            else:
                f = (x - head[1, c]) / head[0, c]
                q = np.where(f <= 1.0, np.rint((f - 0.5) * 65536.0),
                             32768.0 + np.rint((f - 1.0) * 32768.0))
                q = np.clip(q, 0, 65535)
            np.testing.assert_array_equal(rec[:, :, j, c], q.astype(np.uint16))
