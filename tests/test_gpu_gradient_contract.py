"""The one-launch gradient contraction (dftb_gradient_contract) against the two separate entry points on symmetrised
adjoints and atom-block sums, which are held to the oracle elsewhere: atoms of both kinds in any order, block edges (64
atoms per pass), strided adjoints, missing terms, a cutoff, and a molecule whose orbital tables exceed shared memory.

Both sides add the same terms in another order: the tolerance is (terms per atom) 2^-50 of the sum of their absolute
values, which the separate entry points give for absolute adjoints only up to sign, so it is taken from the largest
adjoint and derivative instead."""
import pytest
import torch

from dftbaby_b200 import gradients, native
from dftbaby_b200.params import Parametrization
from test_gpu_sk_tiles import _atoms

pytestmark = pytest.mark.gpu

R_LR = 3.03


class _Mol:
    def __init__(self, al, cutoff):
        dev = torch.device("cuda", 0)
        p = self.par = Parametrization([1, 6])
        ind, ls, ms = [], [], []
        for i, (Z, _) in enumerate(al):
            for (n, l, m) in p.valorbs[Z]:
                ind.append(i)
                ls.append(l)
                ms.append(m)
        i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=dev)
        self.ind, self.ls, self.ms = i32(ind), i32(ls), i32(ms)
        self.atype = i32([p.atom_type[Z] for Z, _ in al])
        self.typ = self.atype[self.ind.long()].contiguous()
        self.sigma = torch.tensor([p.sigmas[Z] for Z, _ in al], dtype=torch.float64, device=dev)
        self.pos = torch.tensor([q for _, q in al], dtype=torch.float64, device=dev).reshape(-1, 3).contiguous()
        n = len(al)
        self.dircos = tuple(torch.empty((n, n), dtype=torch.float64, device=dev) for _ in range(4))
        native.call("dftb_directional_cosines", n, native.ptr(self.pos), *[native.ptr(t) for t in self.dircos],
                    native.stream())
        self.mprox = (self.dircos[0] < cutoff).to(torch.int32)
        self.mprox.fill_diagonal_(1)


def _separate(g, XS, XH, Yg, Ylr, vrep):
    P, st, p = native.ptr, native.stream(), g.par
    nat, norb = g.pos.shape[0], g.ind.shape[0]
    t = p.device_tables(g.pos.device)
    out = torch.zeros(3 * nat, dtype=torch.float64, device=g.pos.device)
    sym = lambda X: None if X is None else (X + X.T).contiguous()
    if XS is not None or XH is not None:
        xs, xh, o = sym(XS), sym(XH), torch.empty_like(out)
        native.call("dftb_sk_gradient_contract", norb, nat, P(g.ind), P(g.typ), P(g.ls), P(g.ms), *[P(q) for q in g.dircos],
                    P(g.mprox), p.deg, P(t["tab_filled_SH0"]), P(t["S_knots"]), P(t["S_coefs"]), P(t["H_knots"]),
                    P(t["H_coefs"]), p.npair, p.nsk, p.npts, P(xs), P(xh), P(o), st)
        out += o
    ind = g.ind.long()
    blocks = lambda Y: None if Y is None else torch.zeros((nat, nat), dtype=Y.dtype, device=Y.device).index_put_(
        (ind[:, None].expand(norb, norb), ind[None].expand(norb, norb)), Y + Y.T, accumulate=True)
    yg, yl, o = blocks(Yg), blocks(Ylr), torch.empty_like(out)
    native.call("dftb_pair_gradients", nat, P(g.pos), P(g.atype), P(g.sigma), R_LR, P(yg), P(yl),
                P(t["vrep_knots"]) if vrep else None, P(t["vrep_coefs"]), P(t["vrep_dmax"]), p.vrep_nknots, P(o), st)
    return out + o


@pytest.mark.parametrize("n,cutoff,terms", [(1, 30.0, "SHGLV"), (2, 30.0, "SHGLV"), (9, 4.0, "SHGLV"), (40, 30.0, "SH"),
                                            (63, 30.0, "SV"), (65, 30.0, "HG"), (66, 6.0, "LV"), (130, 30.0, "SHGLV")])
def test_matches_the_separate_entry_points(n, cutoff, terms):
    g = _Mol(_atoms(n, n + 1), cutoff)
    norb = g.ind.shape[0]
    gen = torch.Generator(device="cuda").manual_seed(n)
    adj = lambda c: torch.randn((norb, norb + 5), dtype=torch.float64, device="cuda", generator=gen)[:, 2:norb + 2] \
        if c in terms else None
    XS, XH, Yg, Ylr, vrep = adj("S"), adj("H"), adj("G"), adj("L"), "V" in terms
    got = gradients.contract(g, g.par, R_LR, XS, XH, Yg, Ylr, vrep)
    ref = _separate(g, XS, XH, Yg, Ylr, vrep)
    # an atom's gradient has at most 4 norb adjoint terms per matrix, each below 2 max|X| times a derivative of order 1
    # (10 for the repulsive potential)
    big = sum(2.0 * X.abs().max() for X in (XS, XH, Yg, Ylr) if X is not None) + 10.0 * vrep
    assert (got - ref).abs().max() <= 16 * norb * 2.0 ** -50 * big


def test_no_terms_give_zeros():
    g = _Mol(_atoms(5, 1), 30.0)
    assert torch.equal(gradients.contract(g, g.par, R_LR, None, None, None, None, False),
                       torch.zeros(15, dtype=torch.float64, device="cuda"))


def test_orbital_tables_beyond_shared_memory():
    """5000 hydrogens in a chain: 25 kB of tables, read from global memory instead."""
    g = _Mol([(1, (1.4 * i, 0.02 * (i % 7), 0.03 * (i % 5))) for i in range(5000)], 30.0)
    gen = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((5000, 5000), dtype=torch.float64, device="cuda", generator=gen)
    got = gradients.contract(g, g.par, R_LR, X, 0.5 * X, X, None, True)
    ref = _separate(g, X, 0.5 * X, X, None, True)
    assert (got - ref).abs().max() <= 16 * 5000 * 2.0 ** -50 * (5.0 * X.abs().max() + 10.0)
