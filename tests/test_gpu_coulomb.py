"""Coulomb products of few columns (dftb_hermitian_rv, dftb_apbv with lc = 0): the edges of their tiles (64 atom
rows, 32 and 128 pairs, 8 columns, 32 columns per block) against plain FP64 products."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu


def _inputs(nat, nocc, nvirt, m, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    gamma = r(nat, nat)
    return gamma + gamma.T, r(nat, nocc, nvirt), 0.1 + torch.rand((nocc, nvirt), dtype=torch.float64, device="cuda",
                                                                  generator=g), r(nocc * nvirt, m)


def _reference(gamma, q, omega, V, square):
    q2, om = q.reshape(q.shape[0], -1), omega.reshape(-1, 1)
    s = torch.sqrt(om) if square else torch.ones_like(om)
    coul = 4.0 * s * (q2.T @ (gamma @ (q2 @ (s * V))))
    # rounding of the three sums: every term carries at most (nat + nat + nov) eps relative to the same products
    # of absolute values
    mag = 4.0 * s * (q2.abs().T @ (gamma.abs() @ (q2.abs() @ (s * V.abs())))) + om ** (2 if square else 1) * V.abs()
    tol = (2 * q2.shape[0] + q2.shape[1] + 8) * 2.0 ** -53 * mag
    return om ** (2 if square else 1) * V + coul, tol


@pytest.mark.parametrize("nat,nocc,nvirt,m", [
    (1, 1, 1, 1), (2, 1, 7, 3), (63, 5, 13, 8), (64, 8, 16, 9), (65, 3, 43, 16), (31, 31, 33, 17), (33, 127, 1, 24),
    (129, 11, 35, 25), (40, 37, 41, 32), (70, 20, 13, 33), (42, 51, 51, 70)])
def test_products_match_plain_fp64(nat, nocc, nvirt, m):
    gamma, q, omega, V = _inputs(nat, nocc, nvirt, m, nat + 7 * m)
    L = native.load()
    ws = torch.empty(max(256, L.dftb_hermitian_rv_workspace_size(nat, m)), dtype=torch.uint8, device="cuda")
    P = native.ptr
    for square in (True, False):
        U = torch.full_like(V, float("nan"))
        if square:
            native.call("dftb_hermitian_rv", nat, nocc, nvirt, m, P(gamma), P(q), P(omega), P(V), P(U), P(ws),
                        ws.numel(), native.stream())
        else:
            native.call("dftb_apbv", nat, nocc, nvirt, m, 0, P(gamma), None, None, P(q), None, P(omega), P(V), P(U),
                        P(ws), ws.numel(), native.stream())
        ref, tol = _reference(gamma, q, omega, V, square)
        assert torch.all((U - ref).abs() <= tol)


def test_operands_off_the_16_byte_grid():
    """Rows of q_ov, V and the outputs may start on any 8-byte boundary."""
    nat, nocc, nvirt, m = 37, 9, 11, 5
    gamma, q, omega, V = _inputs(nat, nocc, nvirt, m, 3)

    def shifted(t):
        buf = torch.zeros(t.numel() + 1, dtype=t.dtype, device=t.device)
        buf[1:] = t.reshape(-1)
        return buf[1:].view(t.shape)

    q, V, omega, gamma = shifted(q), shifted(V), shifted(omega), shifted(gamma)
    U = shifted(torch.zeros_like(V))
    ws = torch.empty(native.load().dftb_hermitian_rv_workspace_size(nat, m), dtype=torch.uint8, device="cuda")
    P = native.ptr
    native.call("dftb_hermitian_rv", nat, nocc, nvirt, m, P(gamma), P(q), P(omega), P(V), P(U), P(ws), ws.numel(),
                native.stream())
    ref, tol = _reference(gamma, q, omega, V, True)
    assert torch.all((U - ref).abs() <= tol)
