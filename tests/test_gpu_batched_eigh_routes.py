"""Batched eigensolver on both sides of the line between its own kernel and the batched library call: residual, orthogonality
and eigenvalues within 30 n ulp of the norm, and an error for a matrix that is not finite."""
import math

import pytest
import torch

from dftbaby_b200 import batched
from dftbaby_b200.exceptions import ExcitedStatesError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 9])
@pytest.mark.parametrize("more", [0, 1])
def test_line(n, more):
    many = batched._many(n)
    B = 1800 + more if many == float("inf") else many + more
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(B, n, n, dtype=torch.float64, device="cuda", generator=g)
    A = A + A.mT
    w, V = batched.batched_eigh(A)
    want = torch.linalg.eigvalsh(A.cpu()).cuda()
    tol = 30 * n * 2.0 ** -52 * want.abs().amax(-1)
    assert bool(((w - want).abs().amax(-1) <= tol).all())
    assert bool(((A @ V - V * w[:, None, :]).abs().amax((1, 2)) <= tol).all())
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert float((V.mT @ V - eye).abs().max()) <= 30 * n * 2.0 ** -52


def test_not_finite():
    A = torch.eye(4, dtype=torch.float64, device="cuda").repeat(100, 1, 1)
    A[57, 2, 1] = math.nan
    with pytest.raises(ExcitedStatesError):
        batched.batched_eigh(A)
