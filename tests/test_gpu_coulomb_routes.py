"""Coulomb products on both sides of the lines between the kernels and cuBLAS: one odd column block, 24 to 33 columns of many
pairs, and few atoms, against plain FP64 products."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nat,no,nv,m", [(3, 4, 2, 33), (48, 7, 9, 40), (49, 7, 9, 40), (5, 347, 346, 24), (5, 347, 346, 25),
                                         (5, 347, 346, 32), (5, 346, 346, 30), (4, 709, 709, 1), (4, 709, 710, 1),
                                         (3, 707, 707, 1), (4, 709, 709, 2)])
def test_products(nat, no, nv, m):
    g = torch.Generator(device="cuda").manual_seed(nat + 7 * m)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    gamma, q, V = r(nat, nat), r(nat, no * nv), r(no * nv, m)
    omega = 0.1 + torch.rand((no * nv, 1), dtype=torch.float64, device="cuda", generator=g)
    ws = torch.full((native.load().dftb_hermitian_rv_workspace_size(nat, m),), 255, dtype=torch.uint8, device="cuda")
    U, P = torch.full_like(V, float("nan")), native.ptr
    native.call("dftb_apbv", nat, no, nv, m, 0, P(gamma), None, None, P(q), None, P(omega), P(V), P(U), P(ws), ws.numel(),
                native.stream())
    want = omega * V + 4.0 * q.T @ (gamma @ (q @ V))
    # every term of the three nested sums carries at most (2 nat + nov) roundings relative to the same products of
    # absolute values, in either order
    mag = omega * V.abs() + 4.0 * q.abs().T @ (gamma.abs() @ (q.abs() @ V.abs()))
    assert bool(((U - want).abs() <= 2 * (2 * nat + no * nv + 8) * 2.0 ** -53 * mag).all())
