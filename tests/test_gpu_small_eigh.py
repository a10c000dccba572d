"""The one-launch symmetric eigensolver at the edges of its tiles, on spectra that deflate and on scaled matrices: residual,
orthogonality and eigenvalues within 30 n ulp of the norm, the bound by which LAPACK tests its symmetric eigensolvers."""
import math

import pytest
import torch

from dftbaby_b200 import eigen

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -52


def _check(A, w, V, want):
    n = A.shape[-1]
    A, w, V = A.cpu(), w.cpu(), V.cpu()
    scale = float(want.abs().max())
    if scale == 0.0:
        scale = 1.0
    # scaled, so that the products of the check neither over- nor underflow
    A, w, want = A / scale, w / scale, want / scale
    tol = 30 * n * ULP
    assert float(torch.linalg.matrix_norm(A @ V - V * w, 2)) <= tol
    assert float(torch.linalg.matrix_norm(V.mT @ V - torch.eye(n, dtype=torch.float64), 2)) <= tol
    assert float((w - want).abs().max()) <= tol
    assert bool((w[1:] >= w[:-1]).all())


def _matrix(kind, n):
    g = torch.Generator().manual_seed(n)
    Q = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, generator=g))[0]
    if kind == "random":
        A = torch.randn(n, n, dtype=torch.float64, generator=g)
    elif kind == "clusters":  # three eigenvalues, all highly degenerate, one split by roundoff
        lam = torch.tensor([1.0, -0.3, 0.5], dtype=torch.float64)[torch.arange(n) % 3]
        A = (Q * (lam + 1e-15 * torch.arange(n))) @ Q.mT
    elif kind == "graded":
        s = 10.0 ** (-12.0 * torch.arange(n, dtype=torch.float64) / n)
        A = torch.randn(n, n, dtype=torch.float64, generator=g)
        A = (A + A.mT) * s[:, None] * s
    elif kind == "wilkinson":  # pairs of eigenvalues that agree to roundoff
        A = torch.diag((torch.arange(n, dtype=torch.float64) - (n - 1) / 2).abs()) + torch.diag(torch.ones(n - 1, dtype=torch.float64), -1)
    elif kind == "blocks":  # decoupled equal blocks: zero off-diagonals in the tridiagonal form
        A = torch.zeros(n, n, dtype=torch.float64)
        for i in range(0, n - 1, 2):
            A[i + 1, i] = 1.0
    elif kind == "diagonal":
        A = torch.diag(torch.randn(n, dtype=torch.float64, generator=g))
    else:
        A = torch.zeros(n, n, dtype=torch.float64)
    return torch.tril(A) + torch.tril(A, -1).mT


@pytest.mark.parametrize("kind", ["random", "clusters", "graded", "wilkinson", "blocks", "diagonal", "zero"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65, 96, 97, 102, 127, 128])
def test_spectra(n, kind):
    A = _matrix(kind, n)
    want = torch.linalg.eigvalsh(A)
    w, V = eigen.eigh(A.cuda())
    _check(A, w, V, want)


@pytest.mark.parametrize("scale", [1e-300, 1e-160, 1e160, 1e300])
def test_scaled(scale):
    A = _matrix("random", 40)
    w, V = eigen.eigh((A * scale).cuda())
    _check(A, w / scale, V, torch.linalg.eigvalsh(A))


@pytest.mark.parametrize("n", [3, 40, 101])
def test_batch_strides_and_triangle(n):
    A = torch.stack([_matrix(k, n) for k in ("random", "clusters", "blocks", "zero", "graded")])
    want = torch.linalg.eigvalsh(A)
    full = torch.full((5, n + 2, n + 3), math.nan, dtype=torch.float64, device="cuda")
    for transpose in (False, True):
        view = full[:, 1:n + 1, 1:n + 1]
        view = view.mT if transpose else view
        view.copy_(torch.where(torch.ones(n, n).tril().bool(), A, torch.tensor(math.nan, dtype=torch.float64)).cuda())
        w, V = eigen.eigh(view)  # the upper triangle is not a number
        for b in range(5):
            _check(A[b], w[b], V[b], want[b])


def test_non_finite_and_dispatch():
    A = torch.stack([_matrix("random", 20) for _ in range(3)]).cuda()
    for bad in (math.nan, math.inf):
        B = A.clone()
        B[1, 7, 3] = bad
        w, V, info = eigen.small_eigh(B)
        assert info.tolist() == [0, 1, 0] and bool(torch.isfinite(w[[0, 2]]).all()) and bool(torch.isnan(w[1]).all())
        with pytest.raises(torch.linalg.LinAlgError):
            eigen.eigh(B)
    big = _matrix("random", eigen.SMALL + 1).cuda()
    w, V = eigen.eigh(big)
    _check(big, w, V, torch.linalg.eigvalsh(big.cpu()))
    X = A[0].clone().requires_grad_()
    eigen.eigh(X)[0].sum().backward()  # torch's own path where a gradient is wanted
    assert torch.allclose(X.grad, torch.eye(20, dtype=torch.float64, device="cuda"))
