"""How many FP32 additions the loss gradient makes to the output layer's bias gradient."""

import pytest
import torch

from pyftle_b200 import _lib
from pyftle_b200._device import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 256, 264, 4096, 10007])
@pytest.mark.parametrize("lddy", [64, 7])
def test_an_addition_per_256_rows_at_most(n, lddy):
    # every row adds 2^-7 (an FP32 and BF16 value) to a sum at 2^24, whose values are 2 apart:
    # an addition of a block's sum is off by at most 1
    y = torch.full((n, 2), 2.0 ** -8 * n, device="cuda")
    target = torch.zeros(n, 2, device="cuda")
    dy = torch.empty(n, lddy, dtype=torch.bfloat16, device="cuda")
    start = torch.full((2,), 2.0 ** 24, device="cuda")
    dbias, loss = start.clone(), torch.zeros(1, device="cuda")
    _lib.call("ftle_mlp_mse_grad", ptr(y), 2, ptr(target), 2, n, ptr(dy), lddy, ptr(dbias),
              ptr(loss), stream_ptr())
    assert torch.equal(dy[:, :2].float(), torch.full((n, 2), 2.0 ** -7, device="cuda"))
    off = (dbias.double() - start.double() - n * 2.0 ** -7).abs().max()
    assert float(off) <= -(-n // 256)
