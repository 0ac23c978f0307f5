"""The FTLE building blocks where their 32-item tiles end, and the 3x3 eigenvalue where its
closed form changes sides or degenerates."""

import numpy as np
import pytest
import torch

from pyftle_b200 import NeighboringParticles
from pyftle_b200.ftle import (
    compute_cauchy_green_2x2,
    compute_cauchy_green_3x3,
    compute_flow_map_jacobian_2x2,
    compute_flow_map_jacobian_3x3,
    compute_ftle_2x2,
    compute_ftle_3x3,
    compute_ftle_from_positions,
    max_eigenvalue_2x2,
    max_eigenvalue_3x3,
)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 1000])
@pytest.mark.parametrize("dim", [2, 3])
def test_blocks_match_numpy_on_ragged_counts(dim, n):
    rng = np.random.default_rng(n)
    K = 2 * dim
    p0 = rng.standard_normal((K * n, dim))
    p1 = rng.standard_normal((K * n, dim))
    part = NeighboringParticles(positions=p0)
    part.positions.copy_(torch.as_tensor(p1))
    a, b = p0.reshape(K, n, dim), p1.reshape(K, n, dim)
    pairs = [(1, 0), (2, 3), (4, 5)][:dim]
    J = np.stack([(b[hi] - b[lo]) / (a[hi] - a[lo])[:, j:j + 1]
                  for j, (hi, lo) in enumerate(pairs)], axis=2)
    jac = (compute_flow_map_jacobian_2x2 if dim == 2 else compute_flow_map_jacobian_3x3)(part)
    np.testing.assert_array_equal(jac.cpu().numpy(), J)
    C = J.transpose(0, 2, 1) @ J if dim == 2 else J @ J.transpose(0, 2, 1)
    cg = (compute_cauchy_green_2x2 if dim == 2 else compute_cauchy_green_3x3)(jac)
    size = np.abs(C).max(axis=(1, 2))
    assert np.all(np.abs(cg.cpu().numpy() - C).max(axis=(1, 2)) <= 8 * 2.0 ** -52 * size)
    lam = np.linalg.eigvalsh(C)[:, -1]
    got = (max_eigenvalue_2x2 if dim == 2 else max_eigenvalue_3x3)(cg).cpu().numpy()
    # the 2D closed form is the reference's, with its cancellation in the discriminant
    np.testing.assert_allclose(got, lam, rtol=1e-7 if dim == 2 else 1e-14)
    want = np.log(np.sqrt(got)) / 2.0
    f = (compute_ftle_2x2 if dim == 2 else compute_ftle_3x3)(jac, 2.0).cpu().numpy()
    np.testing.assert_allclose(f, want, rtol=1e-12, atol=1e-14)
    fused = compute_ftle_from_positions(part, 2.0).cpu().numpy()
    np.testing.assert_allclose(fused, f, rtol=1e-13, atol=1e-15)
    # the planes may also be someone's own tensors
    part.initial_delta_top_bottom = part.initial_delta_top_bottom.clone()
    np.testing.assert_array_equal(compute_ftle_from_positions(part, 2.0).cpu().numpy(), fused)


def _rotated(rng, spectra):
    q = np.linalg.qr(rng.standard_normal((len(spectra), 3, 3)))[0]
    c = (q * spectra[:, None, :]) @ q.transpose(0, 2, 1)
    return 0.5 * (c + c.transpose(0, 2, 1))


@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e140])
def test_max_eigenvalue_3x3_over_spectra(scale):
    rng = np.random.default_rng(4)
    spectra = []
    for gap in (1.0, 1e-2, 1e-6, 1e-10, 1e-15, 0.0):
        r = rng.random((50, 3))
        spectra += [np.stack((1 + 0 * r[:, 0], 1 - gap * r[:, 1], r[:, 2]), 1),      # flat
                    np.stack((1 + 0 * r[:, 0], 0.3 * r[:, 1], 0.3 * r[:, 1] - gap * 0.3), 1),
                    np.stack((1 + gap * r[:, 0], 1 + gap * r[:, 1], 1 + gap * r[:, 2]), 1)]
    spectra += [10.0 ** rng.uniform(-8, 8, (200, 3)), rng.standard_normal((200, 3))]
    C = _rotated(rng, np.concatenate(spectra) * scale)
    C = np.concatenate((C, scale * np.array([np.diag([1.0, 2.0, 3.0]), np.diag([3.0, 2.0, 3.0]),
                                             np.eye(3), np.zeros((3, 3)),
                                             [[0, 1, 0], [1, 0, 0], [0, 0, 0]],
                                             [[1, 1e-170, 0.1], [1e-170, 1, 0], [0.1, 0, 1]],
                                             np.ones((3, 3)), -np.ones((3, 3))])))
    got = max_eigenvalue_3x3(C).cpu().numpy()
    size = np.abs(C).max(axis=(1, 2))
    # LAPACK's own error is a few units of the matrix's size as well
    assert np.all(np.abs(got - np.linalg.eigvalsh(C)[:, -1]) <= 16 * 2.0 ** -52 * size)


def test_max_eigenvalue_3x3_of_matrices_that_are_not_finite():
    C = np.tile(np.eye(3), (6, 1, 1))
    C[0, 0, 0] = np.inf        # a diagonal matrix: its largest element
    C[1, 0, 0] = np.nan
    C[2, 1, 2] = C[2, 2, 1] = np.nan
    C[3, 0, 1] = C[3, 1, 0] = np.inf
    C[4] = np.inf
    C[5] = 2.0 * np.eye(3)
    got = max_eigenvalue_3x3(C).cpu().numpy()
    assert got[0] == np.inf and got[5] == 2.0
    assert np.isnan(got[[2, 3, 4]]).all()
