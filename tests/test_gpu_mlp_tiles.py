"""The MLP GEMM's epilogues where tiles, warps' column groups and work units end."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _call(name, *args):
    from pyftle_b200 import _lib

    _lib.call(name, *args, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


def _bf(shape, gen, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(torch.bfloat16).cuda()


# M: one row group, ragged tiles, more tiles than SMs; N: below, between and past a tile, with
# the column sums' tile changing from unit to unit (three tiles on 148 SMs)
@pytest.mark.parametrize("M,N,K", [(8, 8, 64), (136, 40, 128), (200, 96, 64), (128, 136, 192),
                                   (1000, 384, 64), (148 * 128 + 24, 128, 64),
                                   (60 * 128 + 8, 384, 128)])
def test_epilogues_on_ragged_tiles(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    X, W = _bf((M, K), g), _bf((N, K), g, 0.2)
    b = (torch.randn(N, generator=g) * 0.3).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    pad = 24  # columns past N and rows past M belong to someone else
    acc = X.double() @ W.double().T
    tol = (X.double().abs() @ W.double().abs().T) * K * 2.0 ** -23 + 1e-6

    def out(dtype):
        return torch.full((M + 2, N + pad), 7.0, dtype=dtype, device="cuda")

    def check(t, ref, tol):
        assert torch.all((t[:M, :N].double() - ref).abs() <= tol)
        assert torch.all(t[M:] == 7.0) and torch.all(t[:, N:] == 7.0)

    Z, H, Y = out(torch.float32), out(torch.bfloat16), out(torch.float32)
    _call("ftle_mlp_linear", _p(X), K, _p(W), K, _p(b), M, N, K, 1, _p(Z), N + pad, _p(H), N + pad,
          _p(err))
    _call("ftle_mlp_linear", _p(X), K, _p(W), K, _p(b), M, N, K, 0, _p(Y), N + pad, _p(None), 0,
          _p(err))
    check(Z, acc + b.double(), tol)
    assert torch.equal(Y, Z)
    z = Z[:M, :N].double()
    # sigma's hardware tanh is within 2^-11, the activation rounds to BF16
    check(H, z * torch.sigmoid(z), z.abs() * 2.0 ** -10 + (z * torch.sigmoid(z)).abs() * 2.0 ** -8)
    H2 = out(torch.bfloat16)
    _call("ftle_mlp_linear", _p(X), K, _p(W), K, _p(b), M, N, K, 1, _p(None), 0, _p(H2), N + pad,
          _p(err))
    assert torch.equal(H2, H)

    G, cs = out(torch.bfloat16), torch.full((N,), 0.5, device="cuda")
    _call("ftle_mlp_gemm_dsilu", _p(X), K, 0, _p(W), K, 0, M, N, K, _p(Z), N + pad, _p(G), N + pad,
          _p(cs), _p(err))
    ds = torch.from_numpy(mo.dsilu(z.cpu().numpy())).cuda()
    check(G, acc * ds, acc.abs() * (2.0 ** -9 + z.abs() * 2.0 ** -10) + (acc * ds).abs() * 2.0 ** -8
          + tol * 2.0)
    sums = G[:M, :N].double()
    assert torch.all((cs.double() - 0.5 - sums.sum(0)).abs()
                     <= (sums.abs().sum(0) + 0.5) * M * 2.0 ** -24)
    G2 = out(torch.bfloat16)
    _call("ftle_mlp_gemm_dsilu", _p(X), K, 0, _p(W), K, 0, M, N, K, _p(Z), N + pad, _p(G2), N + pad,
          _p(None), _p(err))
    assert torch.equal(G2, G)
    torch.cuda.synchronize()
    assert int(err.item()) == 0


@pytest.mark.parametrize("splits", [1, 5, 148, 1000])
@pytest.mark.parametrize("M,N", [(8, 64), (264, 136)])
def test_split_k_adds_into_c(M, N, splits):
    g = torch.Generator().manual_seed(splits)
    K = 64 * 37
    A, B = _bf((K, M), g), _bf((K, N), g)
    C = torch.full((M + 1, N + 4), 3.0, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    _call("ftle_mlp_gemm", _p(A), M, 1, _p(B), N, 1, _p(C), N + 4, M, N, K, splits, 1, _p(err))
    ref = 3.0 + A.double().T @ B.double()
    tol = (A.double().abs().T @ B.double().abs() + 3.0) * K * 2.0 ** -23
    assert torch.all((C[:M, :N].double() - ref).abs() <= tol)
    assert torch.all(C[M:] == 3.0) and torch.all(C[:, N:] == 3.0)
    assert int(err.item()) == 0
    assert np.isfinite(C.cpu().numpy()).all()


@pytest.mark.parametrize("outs,lddy,off", [(1, 8, 0), (2, 64, 0), (4, 64, 0), (3, 64, 4), (3, 5, 0)])
@pytest.mark.parametrize("n", [1, 9, 4099])
def test_loss_gradient_rows(n, outs, lddy, off):
    """Wide and single-column stores (a row length or an address that forbids the wide ones)."""
    g = torch.Generator().manual_seed(n + outs)
    y = torch.randn(n, lddy + 2, generator=g).cuda()
    target = torch.randn(n, outs, generator=g).cuda()
    buf = torch.full((off + n * lddy + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    dy = buf[off:]
    db, loss = torch.zeros(4, device="cuda"), torch.zeros(1, device="cuda")
    _call("ftle_mlp_mse_grad", _p(y), lddy + 2, _p(target), outs, n, _p(dy), lddy, _p(db), _p(loss))
    d = y[:, :outs] - target
    got = dy[:n * lddy].view(n, lddy)
    # one FP32 rounding per product, then BF16
    assert torch.all((got[:, :outs].double() - 2.0 * d.double() / n).abs()
                     <= (2.0 * d.double() / n).abs() * 2.0 ** -8)
    assert torch.all(got[:, outs:] == 0.0) and torch.all(buf[off + n * lddy:] == 7.0)
    assert torch.all(buf[:off] == 7.0) and torch.all(db[outs:] == 0.0)
    sums = got[:, :outs].double()
    assert torch.all((db[:outs].double() - sums.sum(0)).abs()
                     <= sums.abs().sum(0) * n * 2.0 ** -24 + 1e-30)
    assert abs(float(loss) - float(d.double().square().sum() / n)) <= n * 2.0 ** -22 * float(
        d.double().square().sum() / n)


def _layered_ftle(net, points, T):
    """The network's FTLE through the layered kernels."""
    _, *jac = net.predict(points, jacobian=True)
    out = torch.empty(points.shape[0], dtype=torch.float64, device="cuda")
    name = "ftle_mlp_jacobian_ftle" if net.dim == 2 else "ftle_mlp_jacobian_ftle3"
    _call(name, *(_p(j) for j in jac), net.OUT_PAD, points.shape[0], ctypes.c_double(net.out_scale),
          ctypes.c_double(T), _p(out))
    return out


# one CTA or two per SM, halves of N = 160 / 192, odd 16-column steps, two feature chunks,
# features wider than the layers, the shallowest and the deepest; tiles are 40 and 32 seeds
@pytest.mark.parametrize("hidden,depth,freqs", [(64, 1, 32), (64, 3, 64), (128, 4, 32), (192, 2, 64),
                                                (256, 4, 32), (256, 8, 32), (320, 2, 32),
                                                (384, 4, 32), (384, 3, 64)])
@pytest.mark.parametrize("dim,n", [(2, 8), (2, 4104), (3, 8), (3, 4104), (2, 20000), (3, 20000)])
def test_fused_field_equals_the_layered_kernels(dim, n, hidden, depth, freqs):
    from pyftle_b200.surrogate import FlowMapMLP, fourier_frequencies

    net = FlowMapMLP(fourier_frequencies(freqs, dim=dim, seed=1), hidden=hidden, depth=depth,
                     out_scale=0.2, seed=2)
    g = torch.Generator(device="cuda").manual_seed(n)
    for l in range(depth + 1):
        net.bias(l)[:net.layers[l].fan_out].normal_(0.0, 0.1, generator=g)
    pts = 6.0 * torch.rand(n, dim + 1, generator=g, dtype=torch.float64, device="cuda")
    ref = _layered_ftle(net, pts, 2.5)
    got = net.ftle(pts, 2.5)
    net.check_errors()
    # the same products in the same order and the same roundings; FP64 at the end
    assert torch.all((got - ref).abs() <= 1e-12 + 1e-9 * ref.abs())
    # changed weights are seen by the next call
    net.wb.mul_(0.5)
    assert torch.all((net.ftle(pts, 2.5) - _layered_ftle(net, pts, 2.5)).abs()
                     <= 1e-12 + 1e-9 * ref.abs().max())


def test_networks_the_fused_field_does_not_take_stay_layered():
    from pyftle_b200 import _lib
    from pyftle_b200.surrogate import FlowMapMLP, fourier_frequencies

    size = _lib.load().ftle_mlp_field_bytes
    for shape in ((2, 448, 4, 32), (2, 512, 4, 32), (3, 256, 9, 32), (2, 256, 4, 96), (4, 256, 4, 32),
                  (2, 96, 4, 32), (2, 256, 0, 32)):
        assert size(*shape) == -1
    assert size(2, 256, 4, 32) == 425984 + 8192
    net = FlowMapMLP(fourier_frequencies(32, dim=3, seed=1), hidden=512, depth=2, out_scale=0.2)
    pts = torch.rand(64, 4, dtype=torch.float64, device="cuda")
    assert torch.equal(net.ftle(pts, 1.0), _layered_ftle(net, pts, 1.0))
