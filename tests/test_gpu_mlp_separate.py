"""The network's element-wise parts one by one (dftb_mlp_bias_relu, dftb_mlp_relu_backward, dftb_mlp_output), which only callers
of the C interface use, at the edges of their 32 x 32 tiles against plain torch.

Tolerances: one FP32 operation each, then rounding to BF16 (2^-8); sums of n FP32 values err by at most n 2^-23 of the sum of
their absolute values."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu
P = native.ptr
BF = torch.bfloat16


def _rand(seed, *shapes):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(s, device="cuda", generator=g) for s in shapes]


@pytest.mark.parametrize("ns,nh", [(1, 1), (31, 33), (32, 32), (65, 40)])
def test_bias_relu_and_backward(ns, nh):
    Z, b, G = _rand(ns, (ns, nh), (nh,), (ns, nh))
    H, HT = torch.full((ns, nh + 1), 7.0, dtype=BF, device="cuda"), torch.full((nh, ns + 2), 7.0, dtype=BF, device="cuda")
    native.call("dftb_mlp_bias_relu", ns, nh, P(Z), nh, P(b), P(H), nh + 1, P(HT), ns + 2, native.stream())
    want = torch.relu(Z + b).to(BF)
    assert torch.equal(H[:, :nh], want) and torch.equal(HT[:, :ns], want.T)
    assert bool((H[:, nh:] == 7.0).all()) and bool((HT[:, ns:] == 7.0).all())
    dZ, dZT = torch.full_like(H, 7.0), torch.full_like(HT, 7.0)
    db = torch.ones(nh, device="cuda")
    native.call("dftb_mlp_relu_backward", ns, nh, P(G), nh, P(H), nh + 1, P(dZ), nh + 1, P(dZT), ns + 2, P(db),
                native.stream())
    masked = torch.where(want > 0, G, torch.zeros_like(G))
    assert torch.equal(dZ[:, :nh], masked.to(BF)) and torch.equal(dZT[:, :ns], masked.to(BF).T)
    s = masked.double()
    assert bool(((db - 1.0 - s.sum(0)).abs() <= (ns + 2) * 2.0 ** -23 * (1.0 + s.abs().sum(0))).all())


@pytest.mark.parametrize("ns,no", [(1, 1), (130, 2), (257, 8)])
def test_output(ns, no):
    Z, b, T, m, wout = _rand(ns + no, (ns, no + 1), (no,), (ns, no), (ns,), (no,))
    Y = torch.empty((ns, no), device="cuda")
    native.call("dftb_mlp_output", ns, no, P(Z), no + 1, P(b), None, None, None, 0.0, P(Y), None, 0, None, 0, None, None,
                native.stream())
    assert torch.equal(Y, Z[:, :no] + b)
    dY, dYT = torch.zeros((ns, no), dtype=BF, device="cuda"), torch.zeros((no, ns), dtype=BF, device="cuda")
    db, loss = torch.zeros(no, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    native.call("dftb_mlp_output", ns, no, P(Z), no + 1, P(b), P(T), P(m), P(wout), 0.5, P(Y), P(dY), no, P(dYT), ns, P(db),
                P(loss), native.stream())
    d = (Y - T).double()
    w = wout.double() * m.double()[:, None]
    g = w * d  # 2 w d / 2
    assert bool(((dY.double() - g).abs() <= (2.0 ** -8 + 2.0 ** -21) * g.abs()).all()) and torch.equal(dY.T, dYT)
    assert bool(((db - g.sum(0)).abs() <= (ns + 8) * 2.0 ** -23 * g.abs().sum(0)).all())
    terms = 0.5 * w * d * d
    assert abs(float(loss) - float(terms.sum())) <= 2.0 ** -21 * float(terms.abs().sum())
