"""How a weight gradient's contraction over the batch is split (no GPU)."""

import pytest

from pyftle_b200.surrogate import _weight_grad_splits


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 6, 9, 16, 36, 64, 149])
def test_pieces_are_short_and_fill_whole_turns(tiles):
    for n in (64, 128, 960, 1024, 1088, 4096, 30016, 65536, 75776, 75840, 1 << 20):
        splits = _weight_grad_splits(n, tiles, 148)
        chunks = n // 64
        piece = -(-chunks // min(splits, chunks)) * 64  # rows, as the GEMM rounds them
        assert piece <= 1024
        turn = max(1, 148 // tiles)
        assert splits % turn == 0 and (splits == turn or n > 1024 * (splits - turn))
