"""Snapshot packing against numpy, at the sizes where its runs, tiles and ranges end."""

import numpy as np
import pytest

from pyftle_b200 import GridSpec, SnapshotSeries

pytestmark = pytest.mark.gpu


def _successors(snaps, periodic_time):
    last = snaps[:1] if periodic_time else snaps[-1:]
    return np.concatenate((snaps[1:], last))


def _bf16(x):
    """Codes of the bfloat16 values nearest to normal float64 x (ties to even, one rounding)."""
    u = np.ascontiguousarray(x).view(np.uint64)
    u = (u + (np.uint64((1 << 44) - 1) + ((u >> np.uint64(45)) & np.uint64(1)))) >> np.uint64(45)
    f = (u << np.uint64(45)).view(np.float64).astype(np.float32)
    return (f.view(np.uint32) >> np.uint32(16)).astype(np.uint16)


@pytest.mark.parametrize("periodic_time", [False, True])
@pytest.mark.parametrize("num", [1, 3, 4, 7, 8, 9, 17])
@pytest.mark.parametrize("shape", [(2, 2), (31, 9), (17, 16), (64, 33), (2, 2, 2), (9, 9, 7)])
def test_packed_records(shape, num, periodic_time):
    dim, nodes = len(shape), int(np.prod(shape))
    rng = np.random.default_rng(num)
    snaps = rng.standard_normal((num, dim, nodes)) * 3.0 + 0.5
    snaps[num // 2, :, nodes // 2] = 0.0
    snaps[-1, 0, -1] = -0.0
    grid = GridSpec(shape, (0.0,) * dim, (1.0,) * dim)
    nxt = _successors(snaps, periodic_time)

    f64 = SnapshotSeries(grid, snaps, precision="fp64", periodic_time=periodic_time)
    got = f64.packed.cpu().numpy().view(np.float64).reshape(num, nodes, 2 * dim)
    np.testing.assert_array_equal(got, np.concatenate((snaps, nxt), axis=1).transpose(0, 2, 1))

    half = 2 if dim == 2 else 4

    def records(precision):
        p = SnapshotSeries(grid, snaps, precision=precision, periodic_time=periodic_time).packed
        raw = p.cpu().numpy()
        rec = raw[256:].view(np.uint16).reshape(num, nodes, 2, half)
        return raw[:64].view(np.float32).reshape(4, 4), rec

    def expect(encode):
        want = np.zeros((num, nodes, 2, half), np.uint16)
        for c in range(dim):
            for j, x in enumerate((snaps, nxt)):
                want[:, :, j, c] = encode(c, x[:, c])
        return want

    _, rec = records("fp16")
    np.testing.assert_array_equal(rec, expect(lambda c, x: x.astype(np.float16).view(np.uint16)))
    _, rec = records("bf16")
    np.testing.assert_array_equal(rec, expect(lambda c, x: _bf16(x)))

    head, rec = records("fx15")
    vmin = np.float64(head[2, :dim])
    step = np.float64(head[3, :dim]) - vmin
    lo = snaps.min(axis=(0, 2))
    assert np.all(vmin <= lo) and np.all(vmin >= np.nextafter(lo.astype(np.float32), -np.inf))
    with np.errstate(divide="ignore", invalid="ignore"):
        np.testing.assert_array_equal(rec, expect(
            lambda c, x: np.clip(np.rint((x - vmin[c]) * (32767 / step[c])), 0, 32767)
            if step[c] > 0 else np.zeros_like(x)))

    head, rec = records("fx16")
    scale, off = head[0].astype(np.float64), head[1].astype(np.float64)

    def fx16(c, x):
        if not scale[c] > 0:
            return np.zeros_like(x)
        f = (x - off[c]) / scale[c]
        q = np.where(f <= 1.0, np.rint((f - 0.5) * 65536.0), 32768.0 + np.rint((f - 1.0) * 32768.0))
        return np.clip(q, 0, 65535)

    np.testing.assert_array_equal(rec, expect(fx16))


@pytest.mark.parametrize("precision", ["fx15", "fx16"])
def test_packing_of_values_that_are_not_finite(precision):
    """A NaN takes code 0 and leaves the range and the other codes alone; an infinity makes the
    range infinite, whose codes are all 0."""
    rng = np.random.default_rng(2)
    grid = GridSpec((40, 30), (0.0, 0.0), (1.0, 1.0))
    snaps = rng.standard_normal((9, 2, 1200))
    ref = SnapshotSeries(grid, snaps, precision=precision).packed.cpu().numpy()
    bad = snaps.copy()
    inner = np.argsort(snaps[4, 0])[600]  # not the range's end
    bad[4, 0, inner] = np.nan
    got = SnapshotSeries(grid, bad, precision=precision).packed.cpu().numpy()
    np.testing.assert_array_equal(got[:256], ref[:256])
    a, b = (x[256:].view(np.uint16).reshape(9, 1200, 2, 2) for x in (got, ref))
    changed = np.argwhere(a != b)
    assert {tuple(i) for i in changed} <= {(4, inner, 0, 0), (3, inner, 1, 0)}
    assert a[4, inner, 0, 0] == 0 and a[3, inner, 1, 0] == 0
    bad[4, 0, inner] = np.inf
    got = SnapshotSeries(grid, bad, precision=precision).packed.cpu().numpy()
    rec = got[256:].view(np.uint16).reshape(9, 1200, 2, 2)
    assert not rec[..., 0].any()
    np.testing.assert_array_equal(rec[..., 1], b[..., 1])
