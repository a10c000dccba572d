"""The small eigensolver on matrices whose secular roots lie on the middle between two poles, where the bracket of the
iteration starts: tridiagonals and dense matrices of small integers, symmetric chains and rings, Clement matrices.  Residual,
orthogonality and eigenvalues within 30 n ulp of the norm, as for the other spectra."""
import numpy as np
import pytest
import torch

from dftbaby_b200 import eigen

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -52


def _check(A):
    """A: (batch, n, n), symmetric, on the CPU."""
    n = A.shape[-1]
    w, V, info = eigen.small_eigh(A.cuda())
    assert not bool(info.any())
    w, V = w.cpu(), V.cpu()
    want = torch.linalg.eigvalsh(A)
    tol = 30 * n * ULP * want.abs().amax(-1).clamp_min(1e-300)
    assert bool(((w - want).abs().amax(-1) <= tol).all())
    assert bool((torch.linalg.matrix_norm(A @ V - V * w[:, None, :], 2) <= tol).all())
    assert float(torch.linalg.matrix_norm(V.mT @ V - torch.eye(n, dtype=A.dtype), 2).max()) <= 30 * n * ULP


def _tridiagonal(d, e):
    d, e = torch.as_tensor(d, dtype=torch.float64), torch.as_tensor(e, dtype=torch.float64)
    return torch.diag_embed(d) + torch.diag_embed(e, -1) + torch.diag_embed(e, 1)


def test_order_five():
    _check(_tridiagonal([[-3, 2, 3, 3, 0]], [[2, -2, 2, -2]]))


@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8, 12])
def test_integer_tridiagonals(n):
    rng = np.random.default_rng(n)
    _check(_tridiagonal(rng.integers(-3, 4, (4000, n)), rng.integers(-2, 3, (4000, n - 1))))


@pytest.mark.parametrize("n", [3, 5, 8, 17])
def test_integer_matrices(n):
    rng = np.random.default_rng(n)
    A = torch.as_tensor(rng.integers(-2, 3, (1000, n, n)), dtype=torch.float64)
    _check(A + A.mT)


@pytest.mark.parametrize("n", [6, 10, 20, 32, 33, 63, 64, 65, 96, 100, 127, 128])
def test_chains_rings_and_clement(n):
    ones = np.ones(n - 1)
    ring = _tridiagonal(np.zeros(n), -ones)
    ring[0, -1] = ring[-1, 0] = -1.0
    k = np.arange(1, n)
    _check(torch.stack([_tridiagonal(np.zeros(n), -ones), ring,
                        _tridiagonal(np.zeros(n), -1.0 + 0.2 * (-1.0) ** k),        # a chain of alternating bonds
                        _tridiagonal(0.5 * (-1.0) ** np.arange(n), ones),           # alternating sites
                        _tridiagonal(np.zeros(n), np.sqrt(k * (n - k)))]))          # eigenvalues n - 1, n - 3, ...


def test_status_is_raised(monkeypatch):
    A = torch.eye(4, dtype=torch.float64, device="cuda")
    for code, words in ((1, "non-finite"), (2, "converge")):
        monkeypatch.setattr(eigen, "small_eigh", lambda M, code=code: (
            M.diagonal(), M, torch.tensor([code], dtype=torch.int32, device="cuda")))
        with pytest.raises(torch.linalg.LinAlgError, match=words):
            eigen.eigh(A)
