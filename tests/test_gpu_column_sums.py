"""How many FP32 additions the backward GEMM makes to a bias gradient."""

import pytest
import torch

from pyftle_b200 import _lib
from pyftle_b200._device import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 72, 128, 200, 256, 384, 520])
@pytest.mark.parametrize("M", [8, 128, 136, 1000, 4104, 30016])
def test_an_addition_per_128_rows_at_most(M, N):
    # A B^T is 2^-5 everywhere and silu'(0) = 1/2, so every row adds 2^-6 (exact in BF16 and
    # FP32) to sums at 2^24, whose values are 2 apart: an addition is off by at most 1
    A = torch.zeros(M, 64, dtype=torch.bfloat16, device="cuda")
    B = torch.zeros(N, 64, dtype=torch.bfloat16, device="cuda")
    A[:, 3], B[:, 3] = 1.0, 2.0 ** -5
    Z = torch.zeros(M, N, device="cuda")
    G = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    sums = torch.full((N,), 2.0 ** 24, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("ftle_mlp_gemm_dsilu", ptr(A), 64, 0, ptr(B), 64, 0, M, N, 64, ptr(Z), N, ptr(G), N,
              ptr(sums), ptr(err), stream_ptr())
    assert torch.equal(G.float(), torch.full((M, N), 2.0 ** -6, device="cuda"))
    off = (sums.double() - 2.0 ** 24 - M * 2.0 ** -6).abs().max()
    assert float(off) <= -(-M // 128)
    assert int(err) == 0
