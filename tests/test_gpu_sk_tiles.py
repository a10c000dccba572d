"""S, H0 and dipoles at the edges of their 8 x 32 atom tiles: atoms of both kinds in any order, partial tiles, a
proximity cutoff inside the molecule, orbitals with l > 1, and tables that do not share their knots."""
import numpy as np
import pytest
import torch

from dftbaby_b200 import native
from dftbaby_b200.dftb2 import DFTB2
from oracle import dftb_oracle as O

pytestmark = pytest.mark.gpu


def _atoms(n, seed):
    """Carbons and hydrogens in random order on a jittered lattice of 2.6 bohr."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    sites = [(i, j, k) for i in range(side) for j in range(side) for k in range(side)][:n]
    Z = [6, 1] + [int(z) for z in rng.choice([1, 6], size=max(0, n - 2))]
    rng.shuffle(Z)
    return [(z, tuple(2.6 * np.array(s) + 0.2 * rng.standard_normal(3))) for z, s in zip(Z[:n], sites)]


@pytest.mark.parametrize("n,cutoff", [(1, 30.0), (2, 30.0), (7, 30.0), (8, 4.0), (9, 30.0), (31, 30.0), (32, 6.0), (33, 30.0),
                                      (65, 8.0)])
def test_matches_oracle(n, cutoff):
    al = _atoms(n, n)
    o = O.DFTB2(al, long_range_correction=0, distance_cutoff=cutoff)
    o.setGeometry(al)
    o._geometry()
    S, H0 = o._constructH0andS()
    o.S = S
    D = o._constructDipoleMatrix()
    g = DFTB2(al, long_range_correction=0, distance_cutoff=cutoff)
    g.setGeometry(al)
    try:
        g._geometry_matrices()
    except torch.linalg.LinAlgError:
        pass  # random atoms: S need not be positive definite; the matrices are formed before its factorisation
    assert np.abs(g.S.cpu().numpy() - S).max() < 1e-13
    assert np.abs(g.H0.cpu().numpy() - H0).max() < 1e-13
    assert np.abs(g.D.cpu().numpy() - D).max() < 1e-12
    assert torch.equal(g.S, g.S.T) and torch.equal(g.H0, g.H0.T)


def _assemble(d, S_tab, H_tab, ls=None):
    """S and H0 of a DFTB2's geometry from given (knots, coefs)."""
    P, t, p = native.ptr, d.par.device_tables(d.device), d.par
    r, x, y, z = d._dircos
    S, H0 = torch.empty_like(d.S), torch.empty_like(d.S)
    native.call("dftb_h0_and_s", d.dim, len(d.atomlist), P(d._ind), P(d._typ), P(d._ls if ls is None else ls), P(d._ms),
                P(r), P(x), P(y), P(z), P(d.Mproximity), P(d._orben), p.deg, P(t["tab_filled_SH0"]), P(S_tab[0]),
                P(S_tab[1]), P(H_tab[0]), P(H_tab[1]), p.npair, p.nsk, p.npts, P(S), P(H0), native.stream())
    return S, H0


def test_tables_with_knots_of_their_own():
    """Each table is evaluated on its own knots: swapping S and H tables swaps the results, and stretching the knots of
    some tables changes those tables' elements only."""
    al = _atoms(20, 5)
    d = DFTB2(al, long_range_correction=0)
    d.setGeometry(al)
    try:
        d._geometry_matrices()
    except torch.linalg.LinAlgError:
        pass
    t = d.par.device_tables(d.device)
    tS, tH = (t["S_knots"], t["S_coefs"]), (t["H_knots"], t["H_coefs"])
    kn = t["H_knots"].clone()
    kn[:, 4:] *= 1.01  # ps and both pp tables
    tX = (kn, t["H_coefs"])
    S, H = _assemble(d, tS, tH)
    off = ~torch.block_diag(*[torch.ones((n, n), dtype=torch.bool, device=S.device) for n in d.orbsPerAtom])
    S2, H2 = _assemble(d, tH, tS)
    assert torch.equal(S2[off], H[off]) and torch.equal(H2[off], S[off])
    SX, HX = _assemble(d, tS, tX)
    XS, _ = _assemble(d, tX, tX)
    assert torch.equal(SX, S) and torch.equal(HX[off], XS[off])
    s_type = d._ls == 0
    ss = s_type[:, None] & s_type[None, :] & off
    assert torch.equal(HX[ss], H[ss]) and not torch.equal(HX[off], H[off])


def test_higher_orbitals_are_nan():
    al = _atoms(10, 3)
    d = DFTB2(al, long_range_correction=0)
    d.setGeometry(al)
    try:
        d._geometry_matrices()
    except torch.linalg.LinAlgError:
        pass
    t = d.par.device_tables(d.device)
    tS, tH = (t["S_knots"], t["S_coefs"]), (t["H_knots"], t["H_coefs"])
    ls = d._ls.clone()
    ls[5] = 2
    S, H = _assemble(d, tS, tH, ls)
    same = d._ind == d._ind[5]
    assert torch.isnan(S[5, ~same]).all() and torch.isnan(H[~same, 5]).all()
    assert not torch.isnan(S[5, same]).any()
    keep = torch.ones(d.dim, dtype=torch.bool, device=S.device)
    keep[5] = False
    assert torch.equal(S[keep][:, keep], d.S[keep][:, keep])
