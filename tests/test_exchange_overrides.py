"""Products of an exchange class whose exchange() or coulomb() is replaced: the replacement's results enter them, and tensors
that it returns keep their values."""
import pytest
import torch

from dftbaby_b200 import native
from dftbaby_b200.lr_tddftb import ExchangeMixed, ExchangeOzaki

NOV, M = 6, 2


def _object(cls):
    x = cls.__new__(cls)
    x.lc, x.products_applied, x.nocc, x.nvirt = 1, 0, 2, 3
    x.omega = 1.0 + torch.arange(NOV, dtype=torch.float64)
    return x


@pytest.fixture
def no_kernels(monkeypatch):
    def refuse(*a):
        raise AssertionError("a kernel was called")

    monkeypatch.setattr(native, "call", refuse)
    monkeypatch.setattr(native, "load", refuse)


@pytest.mark.parametrize("base", [ExchangeMixed, ExchangeOzaki])
@pytest.mark.parametrize("how", ["subclass", "instance", "class"])
def test_replaced_terms(base, how, no_kernels, monkeypatch):
    V = torch.rand(NOV, M, dtype=torch.float64)
    K1, K2, C = torch.rand(NOV, M).double(), torch.rand(NOV, M).double(), torch.rand(NOV, M).double()
    exchange, coulomb = (lambda self, V: (K1, K2)), (lambda self, V: C)
    if how == "subclass":
        x = _object(type("Own", (base,), dict(exchange=exchange, coulomb=coulomb)))
    elif how == "instance":
        x = _object(base)
        x.exchange, x.coulomb = (lambda V: (K1, K2)), (lambda V: C)
    else:
        monkeypatch.setattr(base, "exchange", exchange)
        monkeypatch.setattr(base, "coulomb", coulomb)
        x = _object(base)
    kept = C.clone()
    U, W = x(V)
    assert torch.equal(U, C - K1 - K2) and torch.equal(W, x.omega[:, None] * V + K2 - K1)
    assert torch.equal(C, kept) and x.products_applied == M


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["mixed", "ozaki"])
def test_products_are_those_of_the_terms(name):
    """The products that the solver applies, from one pass, are bit for bit those of exchange() and coulomb(); a strided V
    gives the same."""
    from dftbaby_b200 import LR_TDDFTB, geometry
    al = geometry.polyene(8, sigma=0.02, seed=3)
    td = LR_TDDFTB(al, long_range_correction=1)
    td.setGeometry(al)
    td.dftb2.getEnergy()
    td.setActiveOrbitals(None, None)
    _, q_ov, _ = td._trans_charges(("ov",))
    d = td.dftb2
    occ, virt = (torch.as_tensor(o, device=d.device) for o in (td.active_occupied_orbs, td.active_virtual_orbs))
    omega = (d.orbe[virt][None, :] - d.orbe[occ][:, None]).contiguous()
    Co, Cv = td._active_coefficients()
    cls = ExchangeMixed if name == "mixed" else ExchangeOzaki
    x = cls(d.gamma, d.G_lr, q_ov, omega.reshape(-1), Co, Cv, d.S, len(al), td.nocc, td.nvirt, d.workspace, lc=1)
    g = torch.Generator().manual_seed(0)
    wide = torch.randn(td.nocc * td.nvirt, 7, generator=g, dtype=torch.float64).to(d.device)
    V = wide[:, 1:6:2]
    C, (K1, K2) = x.coulomb(V), x.exchange(V)
    om = omega.reshape(-1)[:, None]
    U, W = x(V)
    # coulomb() sums with atomics, so twice the same call may differ in the last bits
    tol = 64 * 2.0 ** -52 * float(C.abs().max())
    assert float((U - (C - K1 - K2)).abs().max()) <= tol and torch.equal(W, om * V + K2 - K1)
