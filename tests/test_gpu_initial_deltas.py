"""The initial separations that a particle set hands out are the caller's to change."""

import numpy as np
import pytest
import torch

from pyftle_b200.ftle import compute_flow_map_jacobian_2x2, compute_flow_map_jacobian_3x3
from pyftle_b200.particles import NeighboringParticles

pytestmark = pytest.mark.gpu


def _set(dim, n=50):
    p = np.random.default_rng(dim).standard_normal((2 * dim * n, dim))
    part = NeighboringParticles(positions=p)
    part.positions.mul_(1.5)
    return part


@pytest.mark.parametrize("dim", [2, 3])
def test_changing_the_deltas_leaves_the_particles(dim):
    jacobian = compute_flow_map_jacobian_2x2 if dim == 2 else compute_flow_map_jacobian_3x3
    part = _set(dim)
    want, before = jacobian(part), part.initial_delta_right_left.clone()
    deltas = part.initial_deltas()
    deltas.zero_()
    assert torch.equal(part.initial_delta_right_left, before)
    assert torch.equal(part.initial_deltas()[0], before)
    assert torch.equal(jacobian(part), want)


@pytest.mark.parametrize("dim", [2, 3])
def test_replaced_deltas_and_own_ones_are_used(dim):
    jacobian = compute_flow_map_jacobian_2x2 if dim == 2 else compute_flow_map_jacobian_3x3
    part = _set(dim)
    want = jacobian(part)
    part.initial_delta_right_left = 2.0 * part.initial_delta_right_left
    assert torch.equal(jacobian(part)[:, :, 0], 0.5 * want[:, :, 0])

    class Own(NeighboringParticles):
        def initial_deltas(self):
            return 4.0 * super().initial_deltas()

    part = _set(dim)
    part.__class__ = Own
    assert torch.equal(jacobian(part), 0.25 * want)
