"""Largest eigenvalue of 3x3 Cauchy-Green tensors against extended precision, where the
deviation from a multiple of the identity is as small as its rounding, and elsewhere."""

import numpy as np
import pytest
import torch

from pyftle_b200.ftle import max_eigenvalue_3x3

pytestmark = pytest.mark.gpu

N = 4000


def _reference(C):
    """Cyclic Jacobi rotations in numpy's extended precision."""
    a = [[C[:, i, j].astype(np.longdouble) for j in range(3)] for i in range(3)]
    for _ in range(30):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r, apq = 3 - p - q, a[p][q]
            theta = (a[q][q] - a[p][p]) / (2 * np.where(apq == 0, 1, apq))
            t = np.where(theta >= 0, 1, -1) / (np.abs(theta) + np.sqrt(theta * theta + 1))
            t = np.where(apq == 0, 0, t)
            c = 1 / np.sqrt(t * t + 1)
            s = t * c
            a[p][p], a[q][q] = a[p][p] - t * apq, a[q][q] + t * apq
            a[p][q] = a[q][p] = np.zeros_like(apq)
            x, y = a[r][p], a[r][q]
            a[r][p] = a[p][r] = c * x - s * y
            a[r][q] = a[q][r] = s * x + c * y
    return np.maximum(np.maximum(a[0][0], a[1][1]), a[2][2])


def _tensors(kind, size):
    rng = np.random.default_rng(11)
    if kind == "isotropic":
        C = np.eye(3) + size * rng.standard_normal((N, 3, 3))
    else:
        J = rng.standard_normal((N, 3, 3)) * 10.0 ** rng.uniform(-size, size, (N, 1, 3))
        C = J @ np.swapaxes(J, 1, 2)
    return 0.5 * (C + np.swapaxes(C, 1, 2))


@pytest.mark.parametrize("kind,size", [("isotropic", 10.0 ** -k) for k in (16, 15, 14, 11, 8, 2)]
                         + [("stretched", 0), ("stretched", 8)])
def test_largest_eigenvalue(kind, size):
    C = _tensors(kind, size)
    with np.errstate(all="ignore"):
        want = _reference(C)
    got = max_eigenvalue_3x3(torch.as_tensor(C, device="cuda")).cpu().numpy()
    # next to the identity the deviation's error is far below the result's last place: one
    # rounding of it, 2^-53.  Elsewhere the deviation is rounded as often as it is formed from
    # (trace, differences, determinant, two Newton steps): a few 2^-53, as rotations leave
    assert np.max(np.abs((got - want) / want)) < (1.2e-16 if kind == "isotropic" else 4.4e-16)
