"""The FP64 GEMM engine (dftb_dgemm) at the edges of its 64 x 64 x 16 tiles in all operand orders, and the exchange
products in transition-charge form (dftb_apbv / dftb_ambv with lc = 1), whose two-level indices it carries."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (8, 8, 4), (9, 7, 5), (64, 64, 16), (65, 63, 17), (40, 129, 33), (31, 5, 250)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_dgemm_edges(m, n, k, ta, tb):
    g = torch.Generator(device="cuda").manual_seed(m + 5 * n + 11 * k + 2 * ta + tb)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    pad = 3  # leading dimensions beyond the matrix
    A, B, C = r(k, m + pad) if ta else r(m, k + pad), r(n, k + pad) if tb else r(k, n + pad), r(m, n + pad)
    opA = A[:, :m].T if ta else A[:, :k]
    opB = B[:, :k].T if tb else B[:, :n]
    P = native.ptr
    for alpha, beta in ((1.0, 0.0), (-0.75, 0.5)):
        out = C.clone()
        if beta == 0.0:
            out[:, :n] = float("nan")  # not read
        native.call("dftb_dgemm", ta, tb, m, n, k, alpha, P(A), A.stride(0), P(B), B.stride(0), beta, P(out),
                    out.stride(0), native.stream())
        ref = alpha * (opA @ opB) + (beta * C[:, :n] if beta else 0.0)
        tol = 2 * (k + 4) * EPS * (abs(alpha) * (opA.abs() @ opB.abs()) + abs(beta) * C[:, :n].abs())
        assert torch.all((out[:, :n] - ref).abs() <= tol)
        assert torch.equal(out[:, n:], C[:, n:])


@pytest.mark.parametrize("nat,no,nv,m", [(1, 1, 1, 1), (3, 2, 5, 1), (5, 17, 3, 4), (4, 8, 65, 2), (9, 33, 20, 7), (37, 13, 31, 10)])
def test_exchange_in_transition_charge_form(nat, no, nv, m):
    g = torch.Generator(device="cuda").manual_seed(nat + 100 * m)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    sym = lambda X: X + X.transpose(-1, -2)
    gam, glr, q_oo, q_ov, q_vv = sym(r(nat, nat)), sym(r(nat, nat)), sym(r(nat, no, no)), r(nat, no, nv), sym(r(nat, nv, nv))
    omega, v = r(no, nv).abs(), r(no, nv, m)
    L = native.load()
    ws = torch.empty(L.dftb_apbv_workspace_size(nat, no, nv, m), dtype=torch.uint8, device="cuda")
    P = native.ptr

    def parts(f):
        ein = torch.einsum
        coul = 4.0 * ein("Aia,Ac->iac", f(q_ov), f(gam) @ ein("Ajb,jbc->Ac", f(q_ov), f(v)))
        K1 = ein("Bij,Bab,jbc->iac", ein("AB,Aij->Bij", f(glr), f(q_oo)), f(q_vv), f(v))
        K2 = ein("Aib,Aja,jbc->iac", f(q_ov), ein("AB,Bja->Aja", f(glr), f(q_ov)), f(v))
        return omega[:, :, None] * f(v), coul, K1, K2

    omv, coul, K1, K2 = parts(lambda X: X)
    mag = sum(parts(torch.abs))
    # three nested sums of at most nat + no + nv terms each, in two different orders
    tol = 4 * (2 * nat + no + nv + no * nv + 8) * EPS * mag
    for name, ref in (("dftb_apbv", omv + coul - K1 - K2), ("dftb_ambv", omv + K2 - K1)):
        U = torch.empty_like(v)
        native.call(name, nat, no, nv, m, 1, P(gam), P(glr), P(q_oo), P(q_ov), P(q_vv), P(omega), P(v), P(U), P(ws),
                    ws.numel(), native.stream())
        assert torch.all((U - ref).abs() <= tol), name
