"""Residues and reconstruction of the int8 FP64 products (csrc/ozaki_gemm.cu) at every number of moduli, at the edges
of the row and column scaling passes, and at row magnitudes beyond what one power-of-two factor can undo."""
import numpy as np
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191]


def _oz():
    native.load()
    from dftbaby_b200 import ozaki
    return ozaki


def _bits(k, nmod):
    return min(53, int(np.floor((sum(np.log2(MODULI[:nmod])) - 1.0 - np.log2(k) - 1e-6) / 2.0)))


@pytest.mark.parametrize("nmod", range(8, 17))
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
def test_every_modulus_count(nmod, ta, tb):
    """Integer entries of b bits enter exactly and the integer product is exact, so only the reconstruction rounds:
    at most one ulp per limb of the result, and one of the reference."""
    oz = _oz()
    m, n, k = 37, 131, 259
    b = _bits(k, nmod)
    rng = np.random.default_rng(nmod)
    A = rng.integers(-(2 ** b) + 1, 2 ** b, (m, k))
    B = rng.integers(-(2 ** b) + 1, 2 ** b, (k, n))
    # entries of the largest magnitude and of one sign, and rows that cancel
    A[0], B[:, 0] = 2 ** b - 1, 2 ** b - 1
    A[1], B[:, 1] = -(2 ** b) + 1, 2 ** b - 1
    A[2, :] = np.where(np.arange(k) % 2 == 0, 2 ** b - 1, -(2 ** b) + 1)
    ref = A.astype(object) @ B.astype(object)
    dev = lambda X, t: (torch.from_numpy(X.T.astype(np.float64).copy()).cuda().T if t
                        else torch.from_numpy(X.astype(np.float64)).cuda())
    C = oz.matmul(dev(A, ta), dev(B, tb), nmod=nmod)
    oz.check_errors(C.device)
    got = C.cpu().numpy()
    for i in range(m):
        for j in range(n):
            assert abs(int(got[i, j]) - ref[i, j]) * 2 ** 53 <= 4 * abs(ref[i, j]), (i, j)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 7), (32, 32, 8), (33, 31, 9), (5, 300, 64), (257, 1, 129)])
def test_scaling_passes_at_their_edges(m, n, k):
    """Fewer columns than CTAs of the column pass, partial 32-row blocks, one row: against the rounding bound of the
    operands (2^-b of a row's largest entry per entry) and four ulps of the reconstruction."""
    oz = _oz()
    g = torch.Generator().manual_seed(m + 3 * n + 7 * k)
    A = torch.randn(m, k, generator=g, dtype=torch.float64) * 10.0 ** torch.randint(-5, 6, (m, 1), generator=g)
    B = torch.randn(k, n, generator=g, dtype=torch.float64) * 10.0 ** torch.randint(-5, 6, (1, n), generator=g)
    ref = (A.numpy().astype(np.longdouble) @ B.numpy().astype(np.longdouble)).astype(np.float64)
    for ta, tb in ((False, False), (True, False), (False, True), (True, True)):
        a = A.T.contiguous().cuda().T if ta else A.cuda()
        b = B.T.contiguous().cuda().T if tb else B.cuda()
        C = oz.matmul(a, b).cpu().numpy()
        bound = 2.0 ** -53 * (2 * k + 4) * (A.abs().amax(1, keepdim=True) * B.abs().amax(0, keepdim=True)).numpy()
        assert np.all(np.abs(C - ref) <= bound)


@pytest.mark.parametrize("ea,eb", [(900, -880), (-1015, 1000), (1000, 15), (-600, -400)])
def test_extreme_row_scales_are_exact(ea, eb):
    """Rows and columns multiplied by powers of two give the same digits, scaled."""
    oz = _oz()
    g = torch.Generator().manual_seed(2)
    A = torch.rand(40, 70, generator=g, dtype=torch.float64).numpy() + 0.5
    B = torch.rand(70, 50, generator=g, dtype=torch.float64).numpy() + 0.5
    product = lambda X, Y: oz.matmul(torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()).cpu().numpy()
    C, S = product(A, B), product(np.ldexp(A, ea), np.ldexp(B, eb))
    assert np.array_equal(S, np.ldexp(C, ea + eb))
