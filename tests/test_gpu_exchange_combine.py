"""(A+B) V and (A-B) V from the interleaved exchange columns, at the edges of the kernel's blocks: the same bits as the
element-wise passes that the one pass replaces."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("m,nv,no", [(1, 1, 1), (1, 65, 33), (3, 22, 31), (4, 17, 32), (16, 5, 64), (33, 3, 40), (63, 2, 5),
                                     (64, 3, 33), (65, 2, 31), (130, 3, 2)])
def test_blocks(m, nv, no, dtype):
    g = torch.Generator(device="cuda").manual_seed(m * 100 + nv)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)
    Kall, omega, V, U = rnd(m, 2 * nv, no).to(dtype), rnd(no * nv), rnd(no * nv, m), rnd(no * nv, m)
    K = Kall.double().view(m, nv, 2, no).permute(2, 3, 1, 0).reshape(2, no * nv, m)
    want = U - K[0] - K[1], omega[:, None] * V + K[1] - K[0]
    W = torch.empty_like(V)
    native.call("dftb_exchange_combine", m, nv, no, int(dtype == torch.float64), native.ptr(Kall), native.ptr(omega),
                native.ptr(V), native.ptr(U), native.ptr(W), native.stream())
    assert torch.equal(U, want[0]) and torch.equal(W, want[1])
