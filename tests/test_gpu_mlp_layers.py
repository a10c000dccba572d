"""The fused layers of the pair-scoring network (dftb_mlp_inputs, dftb_mlp_dense, dftb_mlp_head) at the edges of their
tiles against plain FP64 on the same BF16 operands.

Tolerances: FP32 accumulation of k products of BF16 operands errs by at most (k + 2) 2^-23 of the sum of their absolute
values; a result stored in BF16 adds 2^-8 of its magnitude."""
import pytest
import torch

from dftbaby_b200 import native, tcgemm

pytestmark = pytest.mark.gpu

P = native.ptr
F32, BF = torch.float32, torch.bfloat16


def _rand(g, *s):
    return torch.randn(s, device="cuda", generator=g)


@pytest.mark.parametrize("ns,nout,nin", [(128, 256, 64), (1, 8, 8), (130, 40, 72), (257, 256, 256), (96, 136, 200)])
@pytest.mark.parametrize("backward", [False, True])
def test_dense_layer(ns, nout, nin, backward):
    native.load()
    g = torch.Generator(device="cuda").manual_seed(ns + nout + nin)
    pad8 = lambda v: (v + 7) // 8 * 8
    X = torch.zeros((ns, pad8(nin)), dtype=BF, device="cuda")
    W = torch.zeros((nout, pad8(nin)), dtype=BF, device="cuda")
    X[:, :nin], W[:, :nin] = _rand(g, ns, nin).to(BF), _rand(g, nout, nin).to(BF)
    bias = _rand(g, nout)
    mask = _rand(g, ns, nout).clamp_min(0.0).to(BF)  # zeros and positive values, as a ReLU leaves
    mask[0, 0] = -0.0
    H, HT = torch.full((ns, nout), 7.0, dtype=BF, device="cuda"), torch.full((nout, ns + 3), 7.0, dtype=BF, device="cuda")
    cs = torch.ones(nout, device="cuda")
    err = tcgemm._errword(X.device)
    native.call("dftb_mlp_dense", ns, nout, nin, P(X), X.stride(0), P(W), W.stride(0), None if backward else P(bias),
                P(mask) if backward else None, nout, P(H), nout, P(HT), ns + 3, P(cs), P(err), native.stream())
    tcgemm.check_errors(X.device)
    x, w = X[:, :nin].double(), W[:, :nin].double()
    V, mag = x @ w.T, x.abs() @ w.abs().T
    tol = (nin + 2) * 2.0 ** -23 * mag
    if backward:
        V, tol = V * (mask.double() > 0), tol * (mask.double() > 0)
    else:
        V, tol = (V + bias.double()).clamp_min(0.0), tol + 2.0 ** -23 * bias.double().abs()
    assert torch.all((H.double() - V).abs() <= tol + 2.0 ** -8 * V.abs() + 1e-30)
    assert torch.equal(HT[:, :ns], H.T) and torch.all(HT[:, ns:] == 7.0)
    assert torch.all((cs.double() - 1.0 - V.sum(0)).abs() <= tol.sum(0) + (ns + 2) * 2.0 ** -23 * (V.abs().sum(0) + 1.0))


@pytest.mark.parametrize("n,ns,nh", [(128, 128, 256), (1, 64, 8), (65, 65, 40), (1000, 1024, 256), (0, 130, 256)])
def test_head(n, ns, nh):
    native.load()
    g = torch.Generator(device="cuda").manual_seed(n + nh)
    H = _rand(g, ns, nh).clamp_min(0.0).to(BF)
    W = _rand(g, 2, nh).to(BF)
    b = _rand(g, 2)
    T, m = _rand(g, n, 2), torch.rand(n, device="cuda", generator=g) + 0.5
    ts, wout = torch.tensor([3.0, 10.0], device="cuda"), torch.tensor([1.0, 0.5], device="cuda")
    msum = m.double().sum() if n else torch.ones((), dtype=torch.float64, device="cuda")
    Y = torch.empty((ns, 2), device="cuda")
    dZ, dZT = torch.empty((ns, nh), dtype=BF, device="cuda"), torch.empty((nh, ns), dtype=BF, device="cuda")
    dW, db, dbz = torch.zeros((2, nh), device="cuda"), torch.zeros(2, device="cuda"), torch.zeros(nh, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    # inference
    native.call("dftb_mlp_head", ns, 0, nh, P(H), nh, P(W), nh, P(b), None, None, None, 0.0, 0.0, None, P(Y), None, 0, None, 0,
                None, None, None, None, native.stream())
    h, w = H.double(), W.double()
    y = h @ w.T + b.double()
    ytol = (nh + 3) * 2.0 ** -23 * (h.abs() @ w.abs().T + b.double().abs())
    assert torch.all((Y.double() - y).abs() <= ytol)
    if n == 0:
        return
    native.call("dftb_mlp_head", ns, n, nh, P(H), nh, P(W), nh, P(b), P(T), P(ts), P(m), 1.0, 0.5, P(msum), None, P(dZ), nh,
                P(dZT), ns, P(dW), P(db), P(dbz), P(loss), native.stream())
    t = (T * ts).double()
    inv = (1.0 / msum.double()).float().double()
    wm = (wout * m[:, None]).double()
    d = y[:n] - t
    gy, gtol = 2.0 * wm * d * inv, 2.0 * wm * inv * (ytol[:n] + 4 * 2.0 ** -23 * d.abs())
    ref = (wm * d * d * inv).sum()
    assert abs(loss.item() - ref.item()) <= (2.0 * wm * inv * d.abs() * ytol[:n]).sum().item() + 2.0 ** -21 * ref.item()
    assert torch.all((db.double() - gy.sum(0)).abs() <= gtol.sum(0) + (n + 2) * 2.0 ** -23 * gy.abs().sum(0))
    # the products take dY rounded to BF16: 2^-9 of it, and the FP32 error before the rounding
    rt = gtol + 2.0 ** -8 * gy.abs()
    hn = h[:n]
    z, zt = (gy @ w) * (hn > 0), (rt @ w.abs()) * (hn > 0)
    assert torch.all((dZ[:n].double() - z).abs() <= zt + 2.0 ** -8 * (z.abs() + zt) + 1e-30)
    assert torch.all(dZ[n:].double() == 0.0) and torch.equal(dZT, dZ.T)
    assert torch.all((dbz.double() - z.sum(0)).abs() <= zt.sum(0) + (n + 2) * 2.0 ** -23 * z.abs().sum(0) + 1e-30)
    sw = gy.T @ hn
    assert torch.all((dW.double() - sw).abs() <= rt.T @ hn.abs() + (n + 2) * 2.0 ** -23 * (gy.abs().T @ hn.abs()) + 1e-30)


@pytest.mark.parametrize("n,ns,nf,ldf", [(1, 128, 8, 8), (63, 64, 8, 9), (65, 128, 3, 3), (200, 256, 8, 8)])
def test_inputs(n, ns, nf, ldf):
    native.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    Fm = _rand(g, n, ldf)
    mean, std = _rand(g, nf), torch.rand(nf, device="cuda", generator=g) + 0.1
    m, msum = torch.rand(n, device="cuda", generator=g), torch.full((1,), 2.0, dtype=torch.float64, device="cuda")
    X, XT = torch.full((ns, 64), 7.0, dtype=BF, device="cuda"), torch.full((64, ns), 7.0, dtype=BF, device="cuda")
    native.call("dftb_mlp_inputs", n, ns, nf, 64, P(Fm), ldf, P(mean), P(std), P(X), 64, P(XT), ns, P(m), P(msum), native.stream())
    assert abs(msum.item() - 2.0 - m.double().sum().item()) <= n * 2.0 ** -50 * (2.0 + m.double().sum().item())
    ref = torch.zeros((ns, 64), dtype=BF, device="cuda")
    ref[:n, :nf] = ((Fm[:, :nf] - mean) / std).to(BF)
    assert torch.equal(X, ref) and torch.equal(XT, ref.T)
