"""The split BF16 GEMM on 256 x 256 tiles of CTA pairs, at the edges of its tiles and K blocks and with every epilogue, against
FP64 and against the 128 x 128 tiles, which add the same products in the same order."""
import pytest
import torch

from dftbaby_b200 import native, tcgemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(129, 1, 8), (256, 256, 64), (257, 255, 65), (300, 513, 15), (511, 257, 129), (640, 300, 200),
                                   (2049, 1025, 49), (4000, 2600, 333)])
@pytest.mark.parametrize("epilogue", ["f32", "pair", "gpt"])
def test_pair_tiles(m, n, k, epilogue):
    native.load()
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    A = torch.randn(m, k, device="cuda", generator=g)
    B = torch.randn(n, k, device="cuda", generator=g)
    G = torch.rand(m, n, device="cuda", generator=g) if epilogue == "gpt" else None
    pa, pb = tcgemm.split(A), tcgemm.split(B)

    def run(wide):
        if epilogue == "f32":
            out = torch.full((m, n), -7.0, device="cuda")
            tcgemm.gemm(pa, pb, K=k, alpha=0.5, out=out, wide=wide, ksplit=1)
            return [out]
        P = tcgemm.Pair(m, n, A.device)
        T = tcgemm.Pair(n, m, A.device) if epilogue == "gpt" else None
        tcgemm.gemm(pa, pb, K=k, alpha=0.5, out_pair=P, wide=wide, **(dict(G=G, out_pair_t=T) if G is not None else {}))
        return [P.hi[:, :n], P.lo[:, :n]] + ([T.hi[:, :m], T.lo[:, :m]] if T is not None else [])

    got, want = run(True), run(False)
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    C = 0.5 * (A.double() @ B.double().T)
    S = 0.5 * (A.double().abs() @ B.double().abs().T)
    if G is not None:
        C, S = C * G, S * G
    val = got[0].double() if epilogue == "f32" else got[0].double() + got[1].double()
    # rounding of both operands to 16 bits and the dropped lo.lo product: below 2^-16 of the sum of absolute products;
    # 3 k additions in FP32, rounding of the result to 16 bits
    assert bool(((val - C).abs() <= (2.0 ** -16 + 3 * k * 2.0 ** -23) * S + 2.0 ** -16 * C.abs()).all())
    if epilogue == "gpt":
        assert torch.equal(got[0].T, got[2]) and torch.equal(got[1].T, got[3])
