"""Error of the weight gradients' contraction over a large batch against FP64."""

import pytest
import torch

from pyftle_b200 import _lib
from pyftle_b200._device import ptr, stream_ptr
from pyftle_b200.surrogate import _weight_grad_splits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out,fan_in", [(64, 256), (256, 256), (384, 384), (512, 512), (1024, 64)])
@pytest.mark.parametrize("n", [960, 16384, 65536])
def test_error_of_the_contraction(n, out, fan_in):
    g = torch.Generator(device="cuda").manual_seed(n + out)
    G = (torch.randn(n, out, device="cuda", generator=g) + 0.2).bfloat16()
    X = (torch.randn(n, fan_in, device="cuda", generator=g) + 0.3).bfloat16()
    W = torch.zeros(out, fan_in, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    splits = _weight_grad_splits(n, -(-out // 128) * -(-fan_in // 128), sms)
    _lib.call("ftle_mlp_gemm", ptr(G), out, 1, ptr(X), fan_in, 1, ptr(W), fan_in, out, fan_in, n,
              splits, 1, ptr(err), stream_ptr())
    want = G.double().T @ X.double()
    # A piece of 1024 rows is 64 additions of 16 products to an FP32 accumulator, which
    # truncates: each loses at most 2^-23 of the sum so far, half of that on average, and the
    # sum so far is half the piece's on average: 64 * 2^-25 = 1.9e-6.  Adding the pieces rounds
    # to nearest, 2^-25 on average each and with either sign: sqrt(72 pieces) * 2^-25 = 2.5e-7.
    assert float((W.double() - want).norm() / want.norm()) < 2.2e-6
    assert int(err) == 0
