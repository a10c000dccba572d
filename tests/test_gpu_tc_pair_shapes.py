"""Shapes that the split BF16 GEMM does send to 256 x 256 tiles of CTA pairs: partial rows and columns, an odd CTA wholly past
the last row, K that ends inside a 64-element block or a 16-element step, the banded order of tall outputs, K ranges that end
half-way through a block; against the 128 x 128 tiles, which add the same products in the same order, and against FP64."""
import pytest
import torch

from dftbaby_b200 import native, tcgemm

pytestmark = pytest.mark.gpu


def _is_pair(m, n, k, ks=1):
    """The rule of the library."""
    cols = -(-n // 256) * ks
    tiles, pairs = -(-m // 128) * cols, -(-m // 256) * cols
    return m > 128 and (tiles > 148 or (tiles >= 80 and k // ks >= 1024)) and 9 * -(-pairs // 74) <= 10 * -(-tiles // 148)


def _operands(m, n, k, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + m + 3 * n + 5 * k)
    A, B = torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g)
    return A, B, torch.rand(m, n, device="cuda", generator=g)


def _bound(A, B, alpha=1.0):
    """Product and error bound of the split: operands rounded to 16 bits and the dropped lo.lo below 2^-16 of the sum of
    absolute products, 3 k additions in FP32, the result rounded to 16 bits."""
    C = alpha * (A.double() @ B.double().T)
    S = abs(alpha) * (A.double().abs() @ B.double().abs().T)
    return C, (2.0 ** -16 + 3 * A.shape[1] * 2.0 ** -23) * S + 2.0 ** -16 * C.abs()


@pytest.mark.parametrize("m,n,k", [(129, 10241, 1025), (256, 10300, 1039), (257, 7000, 1057), (300, 6913, 1024), (511, 5121, 1088),
                                   (385, 6400, 1041), (4100, 2305, 65), (4225, 2049, 17), (4353, 2817, 200), (19001, 255, 33),
                                   (16500, 257, 64), (19000, 1, 100)])
@pytest.mark.parametrize("epilogue", ["f32", "pair", "gpt"])
def test_pairs(m, n, k, epilogue):
    assert _is_pair(m, n, k)
    A, B, G = _operands(m, n, k)
    pa, pb = tcgemm.split(A), tcgemm.split(B)
    outs = []
    for wide in (True, False):
        if epilogue == "f32":
            out = torch.full((m, n), -7.0, device="cuda")
            tcgemm.gemm(pa, pb, K=k, alpha=0.5, out=out, wide=wide, ksplit=1)
            outs.append([out])
            continue
        P, T = tcgemm.Pair(m, n, A.device), tcgemm.Pair(n, m, A.device)
        extra = dict(G=G, out_pair_t=T) if epilogue == "gpt" else {}
        tcgemm.gemm(pa, pb, K=k, alpha=0.5, out_pair=P, wide=wide, **extra)
        outs.append([P.hi[:, :n], P.lo[:, :n]] + ([T.hi[:, :m], T.lo[:, :m]] if extra else []))
    for x, y in zip(*outs):
        assert torch.equal(x, y)
    C, tol = _bound(A, B, 0.5)
    if epilogue == "gpt":
        C, tol = C * G, tol * G
        assert torch.equal(outs[0][0].T, outs[0][2]) and torch.equal(outs[0][1].T, outs[0][3])
    got = outs[0][0].double() if epilogue == "f32" else outs[0][0].double() + outs[0][1].double()
    assert bool(((got - C).abs() <= tol).all())
    tcgemm.check_errors(A.device)


@pytest.mark.parametrize("m,n,k,ks", [(257, 2600, 3168, 3), (511, 2305, 5184, 5), (640, 1000, 6300, 6)])
def test_k_ranges(m, n, k, ks):
    """Ranges of an odd number of 32-element steps: the last block of 64 is half of the next range's."""
    assert _is_pair(m, n, k, ks) and -(-(-(-k // 32)) // ks) % 2 == 1
    A, B, _ = _operands(m, n, k)
    out = torch.full((m, n), -7.0, device="cuda")
    tcgemm.gemm(tcgemm.split(A), tcgemm.split(B), K=k, out=out, wide=True, ksplit=ks)
    C, tol = _bound(A, B)
    assert bool(((out.double() - C).abs() <= tol).all())
    tcgemm.check_errors(A.device)
