"""FP32 outputs of the tensor-core GEMM on rows of every alignment, from every kind of tile, against FP64."""
import pytest
import torch

from dftbaby_b200 import tcgemm

pytestmark = pytest.mark.gpu


def _operands(m, n, k, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + m + 3 * n + 5 * k)
    A, B = torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g)
    return A, B


def _bound(A, B):
    """Product and error bound of the split: operands rounded to 16 bits and the dropped lo.lo below 2^-16 of the sum of
    absolute products, 3 k additions in FP32, the result rounded to 16 bits."""
    C = (A.double() @ B.double().T)
    S = (A.double().abs() @ B.double().abs().T)
    return C, (2.0 ** -16 + 3 * A.shape[1] * 2.0 ** -23) * S + 2.0 ** -16 * C.abs()


@pytest.mark.parametrize("m,n,pad,shift", [(1, 1, 0, 0), (33, 31, 0, 0), (130, 130, 2, 0), (127, 96, 0, 1), (200, 259, 1, 3), (257, 512, 0, 2),
                                           (4100, 2305, 0, 0)])
@pytest.mark.parametrize("mode", ["one pass", "128 x 128", "wide"])
def test_f32_output_rows(m, n, pad, shift, mode):
    """Rows on 4-, 8- and 16-byte boundaries, and nothing written around them."""
    k = 40
    A, B = _operands(m, n, k, 1)
    buf = torch.full((m * (n + pad) + 8,), -7.0, device="cuda")
    out = buf[shift:shift + m * (n + pad)].view(m, n + pad)[:, :n]
    tcgemm.gemm(tcgemm.split(A), tcgemm.split(B), K=k, out=out, refine=mode != "one pass", wide=mode == "wide", ksplit=1)
    if mode == "one pass":
        A, B = A.bfloat16().float(), B.bfloat16().float()
    C, tol = _bound(A, B)
    assert bool(((out.double() - C).abs() <= tol).all())
    out.fill_(-7.0)
    assert bool((buf == -7.0).all())
