"""Blocks per SM of a batch that is given no schedule (no GPU)."""

import math
from types import SimpleNamespace

import pytest

from pyftle_b200.batch import _blocks_per_sm

ITEMS = 9 * 148


def _series(dim, peak, spacing=0.5):
    def peak_speed():
        if peak is None:
            raise AssertionError("not needed here: it waits for the device")
        return peak

    return SimpleNamespace(grid=SimpleNamespace(dim=dim, spacing=(-spacing, 2.0)[:2] + (1.0,) * (dim - 2)),
                           peak_speed=peak_speed)


def _windows(dim, items, steps=10, h=-0.1, count=4):
    share = [items // count] * (count - 1)
    return [SimpleNamespace(positions=SimpleNamespace(shape=(2 * dim * (128 * n - 5), dim)),
                            num_steps=steps, h=h) for n in share + [items - sum(share)]]


def test_3d_and_few_items_take_4_without_a_read_back():
    assert _blocks_per_sm(_series(3, None), _windows(3, 10 * ITEMS)) == 4
    assert _blocks_per_sm(_series(2, None), _windows(2, ITEMS - 1)) == 4
    assert _blocks_per_sm(_series(2, None), _windows(2, 5)) == 4
    assert _blocks_per_sm(_series(2, None), []) == 4


@pytest.mark.parametrize("peak,blocks", [(0.0, 8), (1.0, 8), (500.0, 8), (501.0, 4), (math.inf, 4),
                                         (math.nan, 4)])
def test_many_items_take_8_where_they_stay_compact(peak, blocks):
    # one unit of time at `peak` over cells of 0.5
    assert _blocks_per_sm(_series(2, peak), _windows(2, ITEMS)) == blocks


def test_no_steps():
    assert _blocks_per_sm(_series(2, 1e9), _windows(2, ITEMS, steps=0)) == 8
