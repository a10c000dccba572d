"""What gradients.contract hands to its kernel: FP64 adjoints of (Norb, Norb) on the molecule's device, as rows of a leading
dimension; anything else is refused before a launch."""
import types

import pytest
import torch

from dftbaby_b200 import gradients, native

NAT, NORB = 3, 6


@pytest.fixture
def call(monkeypatch):
    """contract() of a molecule on the CPU; returns the adjoints (XS, XH, Yg, Ylr) that the kernel would read."""
    made, known = [], {}

    def ptr(t):
        if t is None:
            return None
        known[t.data_ptr()] = t
        return t.data_ptr()

    monkeypatch.setattr(native, "ptr", ptr)
    monkeypatch.setattr(native, "stream", lambda: None)
    monkeypatch.setattr(native, "call", lambda name, *a: made.append(a))
    f = lambda *s: torch.zeros(*s, dtype=torch.float64)
    i = lambda *s: torch.zeros(*s, dtype=torch.int32)
    geo = types.SimpleNamespace(ind=i(NORB), typ=i(NORB), ls=i(NORB), ms=i(NORB), dircos=[f(NAT, NAT) for _ in range(4)],
                                mprox=i(NAT, NAT), pos=f(NAT, 3), atype=i(NAT), sigma=f(NAT))
    tables = {k: f(4) for k in ("S_knots", "S_coefs", "H_knots", "H_coefs", "vrep_knots", "vrep_coefs", "vrep_dmax")}
    tables["tab_filled_SH0"] = i(4)
    par = types.SimpleNamespace(device_tables=lambda dev: tables, deg=3, npair=1, nsk=1, npts=1, vrep_nknots=1)

    def run(*adjoints):
        gradients.contract(geo, par, 3.03, *adjoints, False)
        a = made[-1]
        out = []
        for at in (24, 26, 28, 30):
            p, ld = a[at], a[at + 1]
            out.append(None if p is None else known[p].as_strided((NORB, NORB), (ld, 1)))
        return out

    run.made = made
    return run


def _adjoint():
    return torch.rand(NORB, NORB, dtype=torch.float64)


@pytest.mark.parametrize("place", range(4))
@pytest.mark.parametrize("bad", ["smaller", "larger", "not square", "FP32", "another device"])
def test_refused(call, place, bad):
    X = _adjoint()
    X = {"smaller": X[:-1, :-1], "larger": torch.rand(NORB + 1, NORB + 1, dtype=torch.float64), "not square": X[:, :-1],
         "FP32": X.float(), "another device": X.to("meta")}[bad]
    with pytest.raises((RuntimeError, IndexError)):
        call(*[X if k == place else None for k in range(4)])
    assert not call.made


def test_forms(call):
    X = _adjoint()
    wide = torch.rand(NORB, NORB + 3, dtype=torch.float64)[:, 1:NORB + 1]
    column = torch.rand(NORB, 1, dtype=torch.float64)
    for got, want in zip(call(X, X.T, wide, column), (X, X.T, wide, column.expand(NORB, NORB))):
        assert torch.equal(got, want)
    assert call(None, X, None, None)[0] is None
