"""Transition charges at the edges of the kernel's blocks (8 rows, 128 columns), for rows of every alignment and atoms of
one, four and nine orbitals, against the definition in plain FP64 torch."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("nocc,nvirt,shift", [(1, 1, 0), (7, 8, 1), (9, 127, 0), (16, 128, 0), (16, 128, 1), (33, 129, 1),
                                              (130, 257, 0), (257, 31, 1), (64, 384, 0)])
@pytest.mark.parametrize("opa", [(1, 4, 4, 1), (4, 9, 1, 9, 4, 0, 2)])
def test_blocks(nocc, nvirt, shift, opa):
    g = torch.Generator(device="cuda").manual_seed(nocc * 1000 + nvirt)
    opa = list(opa) * 3
    nat, norb = len(opa), sum(opa)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)
    S = rnd(norb, norb)
    S = S + S.mT
    co, cv = rnd(norb, nocc), rnd(norb, nvirt)
    dims = ((nocc, nocc), (nocc, nvirt), (nvirt, nvirt))
    # guard elements on both sides of every output; shift 1: bases off the 16-byte boundary
    bufs = [torch.full((nat * a * b + 4,), -7.0, dtype=torch.float64, device="cuda") for a, b in dims]
    outs = [x[2 - shift:2 - shift + nat * a * b] for x, (a, b) in zip(bufs, dims)]
    L = native.load()
    ws = torch.empty(L.dftb_trans_charges_workspace_size(norb, nocc, nvirt), dtype=torch.uint8, device="cuda")
    ot = torch.tensor(opa, dtype=torch.int32, device="cuda")
    native.call("dftb_trans_charges", norb, nat, nocc, nvirt, native.ptr(co), native.ptr(cv), native.ptr(S),
                native.ptr(ot), *[native.ptr(o) for o in outs], native.ptr(ws), ws.numel(), native.stream())
    for out, buf, (a, b), C1, C2 in zip(outs, bufs, dims, (co, co, cv), (co, cv, cv)):
        S1, S2, A1, A2 = S @ C1, S @ C2, S.abs() @ C1.abs(), S.abs() @ C2.abs()
        got, f = out.view(nat, a, b), 0
        for A, n in enumerate(opa):
            s = slice(f, f + n)
            want = 0.5 * (C1[s].mT @ S2[s] + S1[s].mT @ C2[s])
            # both sides round sums of norb and of 2 n products: at most norb + 2 n + 4 roundings a term each
            bound = 2 * (norb + 2 * n + 4) * EPS * (C1[s].abs().mT @ A2[s] + A1[s].mT @ C2[s].abs())
            assert bool(((got[A] - want).abs() <= bound).all()), (A, n)
            f += n
        assert bool((buf[:2 - shift] == -7.0).all()) and bool((buf[2 - shift + out.numel():] == -7.0).all())


@pytest.mark.parametrize("nat", [1, 31, 511, 512, 513, 1500])
def test_many_atoms(nat):
    """Orbital offsets over several rounds of the scan."""
    opa = [1 + 3 * (i % 3 == 0) for i in range(nat)]
    norb = sum(opa)
    g = torch.Generator(device="cuda").manual_seed(nat)
    co = torch.randn(norb, 3, dtype=torch.float64, device="cuda", generator=g)
    S = torch.eye(norb, dtype=torch.float64, device="cuda")
    q = torch.empty(nat, 3, 3, dtype=torch.float64, device="cuda")
    L = native.load()
    ws = torch.empty(L.dftb_trans_charges_workspace_size(norb, 3, 0), dtype=torch.uint8, device="cuda")
    ot = torch.tensor(opa, dtype=torch.int32, device="cuda")
    native.call("dftb_trans_charges", norb, nat, 3, 0, native.ptr(co), None, native.ptr(S), native.ptr(ot),
                native.ptr(q), None, None, native.ptr(ws), ws.numel(), native.stream())
    ind = torch.repeat_interleave(torch.arange(nat, device="cuda"), ot.long())
    want = torch.zeros_like(q).index_add_(0, ind, co[:, :, None] * co[:, None, :])
    # four products a charge
    assert float((q - want).abs().max()) <= 8 * EPS * float((co.abs().amax() ** 2) * 4)
