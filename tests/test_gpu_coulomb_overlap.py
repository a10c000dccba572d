"""Coulomb products on both sides of the size up to which their kernels overlap: many in a row that feed one another on one
stream, on two streams at once, and captured, against plain FP64 products."""
import pytest
import torch

from dftbaby_b200 import native
from test_gpu_coulomb import _inputs, _reference

pytestmark = pytest.mark.gpu


def _call(gamma, q, omega, V, U, ws):
    nat, nocc, nvirt = q.shape
    P = native.ptr
    native.call("dftb_hermitian_rv", nat, nocc, nvirt, V.shape[1], P(gamma), P(q), P(omega), P(V), P(U), P(ws), ws.numel(),
                native.stream())


@pytest.mark.parametrize("nat,nocc,nvirt,m", [(3, 5, 7, 2), (42, 51, 51, 10), (100, 144, 145, 9), (100, 145, 146, 9)])
def test_chains_streams_and_capture(nat, nocc, nvirt, m):
    gamma, q, omega, V = _inputs(nat, nocc, nvirt, m, nat + m)
    q, gamma = q / (nat * nocc * nvirt) ** 0.5, gamma / nat  # products of order one, so that chains stay finite
    L = native.load()
    size = max(256, L.dftb_hermitian_rv_workspace_size(nat, m))
    ws = [torch.empty(size, dtype=torch.uint8, device="cuda") for _ in range(2)]
    outs = [[torch.empty_like(V) for _ in range(6)] for _ in range(2)]

    def chain(k):
        X = V
        for U in outs[k]:
            _call(gamma, q, omega, X, U, ws[k])  # the next product reads what this one writes
            X = U

    def check(k):
        X = V
        for U in outs[k]:
            ref, tol = _reference(gamma, q, omega, X, True)
            assert torch.all((U - ref).abs() <= tol)
            X = U

    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(2):
        with torch.cuda.stream(streams[k]):
            chain(k)
    torch.cuda.synchronize()
    check(0)
    check(1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(0)
    for U in outs[0]:
        U.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    check(0)
