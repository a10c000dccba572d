"""Long-range corrected products in transition-charge form, their two exchange terms side by side (the workspace that is asked
for) and one after the other (the least that is accepted), at the edges of the tiles and for windows of one orbital, against
plain FP64 products; in a chain, on two streams and in a graph."""
import pytest
import torch

from dftbaby_b200 import native

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _inputs(nat, no, nv, m, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + 1000 * nat + m)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    # neither g_lr nor q_oo and q_vv symmetric, so that no index order is hidden
    return dict(g=r(nat, nat), g_lr=r(nat, nat), q_oo=r(nat, no, no), q_ov=r(nat, no, nv), q_vv=r(nat, nv, nv),
                omega=0.1 + torch.rand((no, nv), dtype=torch.float64, device="cuda", generator=g), V=r(no, nv, m))


def _least(nat, no, nv, m):
    """The workspace of one term at a time."""
    align = lambda n: (n + 255) // 256 * 256
    k1 = nat * no * no + nat * no * nv * m
    k2 = nat * no * nv + nat * nv * nv * m
    return align(8 * max(k1, k2)) + native.load().dftb_hermitian_rv_workspace_size(nat, m)


def _run(name, t, least=False, U=None, ws=None):
    nat, no, nv = t["q_ov"].shape
    m = t["V"].shape[2]
    P = native.ptr
    if ws is None:
        size = _least(nat, no, nv, m) if least else native.load().dftb_apbv_workspace_size(nat, no, nv, m)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    U = torch.full_like(t["V"], float("nan")) if U is None else U
    native.call(name, nat, no, nv, m, 1, P(t["g"]), P(t["g_lr"]), P(t["q_oo"]), P(t["q_ov"]), P(t["q_vv"]), P(t["omega"]),
                P(t["V"]), P(U), P(ws), ws.numel(), native.stream())
    return U


def _reference(name, t):
    """The products and their rounding bound: every term of the nested sums carries at most as many roundings as the sums have
    terms, relative to the same products of absolute values; the kernel and this sum each."""
    def products(t, sign):
        K1 = torch.einsum("Aij,AB,Bab,jbc->iac", t["q_oo"], t["g_lr"], t["q_vv"], t["V"])
        K2 = torch.einsum("Aib,AB,Bja,jbc->iac", t["q_ov"], t["g_lr"], t["q_ov"], t["V"])
        C = 4.0 * torch.einsum("Aia,AB,Bjb,jbc->iac", t["q_ov"], t["g"], t["q_ov"], t["V"]) if name == "dftb_apbv" else 0.0
        return t["omega"][..., None] * t["V"] + C + (-K1 - K2 if name == "dftb_apbv" else sign * -K1 + K2)
    nat, no, nv = t["q_ov"].shape
    terms = 2 * nat + no + nv + nat * max(no, nv) + no * nv + 16
    a = {k: x.abs() for k, x in t.items()}
    K1 = torch.einsum("Aij,AB,Bab,jbc->iac", a["q_oo"], a["g_lr"], a["q_vv"], a["V"])
    K2 = torch.einsum("Aib,AB,Bja,jbc->iac", a["q_ov"], a["g_lr"], a["q_ov"], a["V"])
    C = 4.0 * torch.einsum("Aia,AB,Bjb,jbc->iac", a["q_ov"], a["g"], a["q_ov"], a["V"]) if name == "dftb_apbv" else 0.0
    return products(t, 1.0), 2 * terms * EPS * (a["omega"][..., None] * a["V"] + C + K1 + K2)


@pytest.mark.parametrize("nat,no,nv,m", [(1, 1, 1, 1), (2, 1, 5, 1), (3, 4, 2, 1), (3, 4, 2, 3), (5, 7, 1, 2), (14, 16, 16, 1),
                                         (14, 16, 16, 10), (16, 32, 17, 4), (22, 26, 26, 1), (21, 33, 65, 2), (42, 20, 31, 5)])
@pytest.mark.parametrize("name", ["dftb_apbv", "dftb_ambv"])
def test_products(nat, no, nv, m, name):
    t = _inputs(nat, no, nv, m)
    want, tol = _reference(name, t)
    for least in (False, True):
        got = _run(name, t, least)
        assert bool(((got - want).abs() <= tol).all())


def test_workspace():
    """Less than the least is refused; the size asked for never falls from a smaller call to a larger one."""
    L = native.load()
    t = _inputs(6, 6, 6, 2)
    ws = torch.empty(_least(6, 6, 6, 2) - 1, dtype=torch.uint8, device="cuda")
    for name in ("dftb_apbv", "dftb_ambv"):
        with pytest.raises(native.NativeError, match="workspace"):
            _run(name, t, ws=ws)
    for nat, no, nv in ((14, 16, 16), (62, 76, 76), (82, 101, 101), (90, 111, 111), (336, 609, 609)):
        sizes = [L.dftb_apbv_workspace_size(nat, no, nv, m) for m in range(1, 20)]
        assert sizes == sorted(sizes)
        assert all(s >= _least(nat, no, nv, m) for m, s in enumerate(sizes, 1))


def test_chain_streams_and_graph():
    """Calls that follow one another (each reads the last one's result) with one workspace, on two streams at a time, and
    replayed from a graph."""
    ts = [_inputs(14, 16, 16, 1, 1), _inputs(22, 26, 26, 3, 2)]
    for t in ts:
        t["V"] *= 1e-3
    steps = 6

    def chain(t, bufs, ws):
        for s in range(steps):
            _run(("dftb_apbv", "dftb_ambv")[s % 2], dict(t, V=bufs[s]), U=bufs[s + 1], ws=ws)

    def buffers(t):
        bufs = [torch.zeros_like(t["V"]) for _ in range(steps + 1)]
        bufs[0].copy_(t["V"])
        nat, no, nv = t["q_ov"].shape
        size = native.load().dftb_apbv_workspace_size(nat, no, nv, t["V"].shape[2])
        return bufs, torch.empty(size, dtype=torch.uint8, device="cuda")

    want = []
    for t in ts:
        bufs, ws = buffers(t)
        for s in range(steps):
            _run(("dftb_apbv", "dftb_ambv")[s % 2], dict(t, V=bufs[s]), U=bufs[s + 1], ws=ws)
            torch.cuda.synchronize()
        want.append(bufs[-1].clone())
    close = lambda x, y: float((x - y).abs().max()) <= 1e-11 * float(y.abs().max())  # the order of the atomics varies
    state = [buffers(t) for t in ts]
    streams = [torch.cuda.Stream() for _ in ts]
    torch.cuda.synchronize()
    for _ in range(20):
        for t, (bufs, ws), st in zip(ts, state, streams):
            with torch.cuda.stream(st):
                chain(t, bufs, ws)
    torch.cuda.synchronize()
    for (bufs, _), w in zip(state, want):
        assert close(bufs[-1], w)
    bufs, ws = state[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(ts[0], bufs, ws)
    for _ in range(3):
        for b in bufs[1:]:
            b.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert close(bufs[-1], want[0])
