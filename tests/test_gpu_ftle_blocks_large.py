"""FTLE building blocks on more groups than their blocks cover at once: the shared-memory tiles
are used again, and the results are those of the same groups in small pieces."""

import numpy as np
import pytest
import torch

from pyftle_b200 import ftle as F
from pyftle_b200.particles import NeighboringParticles

pytestmark = pytest.mark.gpu

N = 1_300_003  # the tiles of 9,472 blocks hold 1,212,416 items
PIECE = 100_000


def _calls(dim):
    if dim == 2:
        return (F.compute_flow_map_jacobian_2x2, F.compute_cauchy_green_2x2, F.max_eigenvalue_2x2,
                F.compute_ftle_2x2)
    return (F.compute_flow_map_jacobian_3x3, F.compute_cauchy_green_3x3, F.max_eigenvalue_3x3,
            F.compute_ftle_3x3)


def _particles(first, last):
    part = NeighboringParticles(positions=first)
    part.positions.copy_(last)
    return part


@pytest.mark.parametrize("dim", [2, 3])
def test_large_stacks(dim):
    jacobian, cauchy_green, eigenvalue, ftle = _calls(dim)
    g = torch.Generator(device="cuda").manual_seed(dim)
    kw = dict(dtype=torch.float64, device="cuda", generator=g)
    first = torch.randn(2 * dim, N, dim, **kw)
    last = first + 0.3 * torch.randn(2 * dim, N, dim, **kw)
    part = _particles(first.view(-1, dim), last.view(-1, dim))
    J = jacobian(part)
    C = cauchy_green(J)
    whole = (J, C, eigenvalue(C), ftle(J, 2.0), F.compute_ftle_from_positions(part, 2.0),
             part.initial_delta_top_bottom, part.initial_centroid)
    for a in range(0, N, PIECE):
        b = min(N, a + PIECE)
        p = _particles(first[:, a:b].reshape(-1, dim), last[:, a:b].reshape(-1, dim))
        j = jacobian(p)
        c = cauchy_green(j)
        piece = (j, c, eigenvalue(c), ftle(j, 2.0), F.compute_ftle_from_positions(p, 2.0),
                 p.initial_delta_top_bottom, p.initial_centroid)
        for x, y in zip(whole, piece):
            assert torch.equal(x[a:b], y)
    # a piece itself: J against numpy
    x = last[:, :1000].cpu().numpy()
    d = first[:, :1000].cpu().numpy()
    for k, (plus, minus) in enumerate(((1, 0), (2, 3), (4, 5))[:dim]):
        want = (x[plus] - x[minus]) / (d[plus] - d[minus])[:, k:k + 1]
        np.testing.assert_array_equal(J[:1000, :, k].cpu().numpy(), want)
