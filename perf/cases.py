"""Measured workloads of the framework: single layers of the LR-TD-DFTB path and one whole solve.

Every case calls public entry points (the C ABI through ``native.call``, the product classes, the FP64
product on the int8 tensor cores, the learned network, ``LR_TDDFTB``) at sizes of the repository's benchmark
configurations:

* ``geometry``   -- directional cosines, H0/S, dipoles, gamma and its AO expansion of one geometry: the first
                    step of every solve and of every trajectory step;
* ``gradient``   -- the contraction of a state's adjoint matrices with the spline and pair derivatives: the
                    last step of every excited-state gradient;
* ``charges``    -- Mulliken transition charges q_oo, q_ov, q_vv of an orbital window;
* ``hermitian``  -- one Davidson product R.V without long-range correction;
* ``apbv``       -- (A+B).V and (A-B).V in the transition-charge form of the C interface, long-range corrected;
* ``fp64gemm``   -- an FP64 product of the SCC on the int8 tensor cores;
* ``exact_lc``   -- (A+B).V and (A-B).V with the FP64 exchange on the int8 tensor cores (correction columns);
* ``mixed_lc``   -- the same with the split-BF16 exchange (the Davidson's columns);
* ``train``      -- loss and gradients of the pair-scoring network over one mini-batch (forward and backward);
* ``solve``      -- ``LR_TDDFTB`` of one geometry without long-range correction, from the atom list to the
                    excitation energies and oscillator strengths.

``listed()`` names the sizes, ``draw(rng)`` gives others of the same ranges.  Inputs are made from the seed
alone, on the GPU.  ``exact()`` restates each layer in plain FP64 torch.
"""
import math

import torch

from dftbaby_b200 import geometry, gradients, learned, lr_tddftb, native, ozaki
from dftbaby_b200.params import Parametrization

R_LR = 3.03       # long-range radius (bohr), the framework's default
CUTOFF = 30.0     # distance cutoff of the Slater-Koster elements (bohr)


def listed():
    return [
        # C20H22, the plain TD-DFTB benchmark molecule: the smallest call, where launches count
        dict(name="geometry-c20h22", op="geometry", shape="polyene", n=20),
        # C1014H90, the 1104-atom benchmark flake: 4146 orbitals
        dict(name="geometry-c1014h90", op="geometry", shape="armchair", n=7),
        # C40H42, the trajectory benchmark's molecule: one gradient per time step
        dict(name="gradient-c40h42", op="gradient", shape="polyene", n=40, lc=True),
        # a held-out flake of the learned-start benchmark with its full window, C294H42 (odd row lengths)
        dict(name="charges-c294h42", op="charges", shape="flake", n=7, nocc=609, nvirt=609),
        # ten states of C20H22: 42 atoms, 51 x 51 pairs
        dict(name="hermitian-c20h22", op="hermitian", shape="polyene", n=20, nocc=51, nvirt=51, m=10),
        # ten states of C294H42 over its 371k pairs
        dict(name="hermitian-c294h42", op="hermitian", shape="flake", n=7, nocc=609, nvirt=609, m=10),
        # the drop-in (A+B).v / (A-B).v calls for five states (ten vectors) of C40H42
        dict(name="apbv-c40h42", op="apbv", shape="polyene", n=40, nocc=101, nvirt=101, m=10),
        # the SCC's Norb^3 product at 4146 orbitals
        dict(name="fp64gemm-4146", op="fp64gemm", rows=4146, cols=4146, inner=4146),
        # correction columns of the 1104-atom benchmark, window 1225 x 1225
        dict(name="exact-lc-c1014h90", op="exact_lc", shape="armchair", n=7, nocc=1225, nvirt=1225, m=4),
        # Davidson columns of the 1104-atom benchmark, window 1225 x 1225
        dict(name="mixed-lc-c1014h90", op="mixed_lc", shape="armchair", n=7, nocc=1225, nvirt=1225, m=16),
        # one mini-batch of the network's training
        dict(name="train-65536", op="train", samples=65536),
        # ten states of C20H22, the plain TD-DFTB benchmark, start to finish
        dict(name="solve-c20h22", op="solve", shape="polyene", n=20, nstates=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_molecule(rng, largest_flake=7):
    """A polyene, acene or flake: 12 to 1104 atoms."""
    shape = rng.choice(["polyene", "acene", "flake", "armchair"])
    n = {"polyene": 2 * rng.randint(3, 30), "acene": rng.randint(2, 8), "flake": rng.randint(2, largest_flake),
         "armchair": rng.randint(1, 4)}[shape]
    return dict(shape=shape, n=n)


def draw(rng):
    op = rng.choice(["geometry", "gradient", "charges", "hermitian", "apbv", "fp64gemm", "exact_lc", "mixed_lc",
                     "train", "solve"])
    if op == "geometry":
        return dict(op=op, **_draw_molecule(rng, 12))
    if op == "gradient":
        return dict(op=op, lc=rng.random() < 0.75, **_draw_molecule(rng))
    if op in ("charges", "hermitian", "exact_lc", "mixed_lc"):
        mol = _draw_molecule(rng)
        norb = _norb(mol)
        half = norb // 2
        # full and truncated windows, odd and even
        nocc, nvirt = _log_int(rng, max(8, half // 4), half), _log_int(rng, max(8, half // 4), half)
        case = dict(op=op, nocc=nocc, nvirt=nvirt, **mol)
        if op != "charges":
            case["m"] = _log_int(rng, 1, 4 if op == "exact_lc" else 30)
        return case
    if op == "apbv":
        n = 2 * rng.randint(3, 22)
        half = (5 * n + 2) // 2
        return dict(op=op, shape="polyene", n=n, nocc=rng.randint(half // 2, half), nvirt=rng.randint(half // 2, half),
                    m=_log_int(rng, 1, 10))
    if op == "fp64gemm":
        norb = _log_int(rng, 100, 4146)
        return dict(op=op, rows=rng.choice([norb, norb // 2]), cols=rng.choice([norb, norb // 2]), inner=norb)
    if op == "train":
        return dict(op=op, samples=_log_int(rng, 1000, 65536))
    shape = rng.choice(["polyene", "acene"])
    return dict(op=op, shape=shape, n=2 * rng.randint(4, 20) if shape == "polyene" else rng.randint(2, 8),
                nstates=rng.randint(3, 12))


# ---------------------------------------------------------------- inputs
def _molecule(case, seed):
    """Seeded distorted molecule of the case (Angstrom noise as in the benchmark configurations)."""
    build = dict(polyene=geometry.polyene, acene=geometry.acene, flake=geometry.hexagonal_flake,
                 armchair=geometry.armchair_flake)[case["shape"]]
    return build(case["n"], sigma=0.02, seed=seed)


def _norb(case):
    return sum(4 if Z == 6 else 1 for Z, _ in _molecule(case, 0))


class _Tables:
    """The orbital and atom tables of one molecule and the parameter tables, as a solver object holds them."""

    def __init__(self, mol, dev):
        p = self.par = Parametrization([1, 6])
        self.tables = p.device_tables(dev)
        ind, ls, ms, orben = [], [], [], []
        for i, (Z, _) in enumerate(mol):
            for (n, l, m) in p.valorbs[Z]:
                ind.append(i)
                ls.append(l)
                ms.append(m)
                orben.append(p.orbital_energies[Z][(n, l)])
        Zs = [Z for Z, _ in mol]
        i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=dev)
        f64 = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
        self.nat, self.norb = len(mol), len(ind)
        self.ind, self.ls, self.ms, self.orben = i32(ind), i32(ls), i32(ms), f64(orben)
        self.atype = i32([p.atom_type[Z] for Z in Zs])
        self.typ = self.atype[self.ind.long()].contiguous()
        self.opa = i32([len(p.valorbs[Z]) for Z in Zs])
        self.sigma = f64([p.sigmas[Z] for Z in Zs])
        self.pos = f64([q for _, q in mol]).reshape(-1, 3).contiguous()
        self.mprox = None


def _distances(pos):
    """(r, x, y, z) of slako.directional_cosines in plain torch."""
    d = pos[:, None, :] - pos[None, :, :]
    r = torch.sqrt((d * d).sum(-1))
    e = d / torch.where(r > 0.0, r, torch.ones_like(r))[..., None]
    e[r == 0.0] = torch.tensor([0.0, 0.0, 1.0], dtype=e.dtype, device=e.device)
    return r, e[..., 0].contiguous(), e[..., 1].contiguous(), e[..., 2].contiguous()


def _mprox(r):
    m = (r < CUTOFF).to(torch.int32)
    m.fill_diagonal_(1)
    return m


def _gamma(r, sigma, extra):
    """erf(R / sqrt(2 (sA^2 + sB^2 + extra))) / R with its on-site limit."""
    s2 = sigma[:, None] ** 2 + sigma[None, :] ** 2 + extra
    off = torch.erf(r / torch.sqrt(2.0 * s2)) / torch.where(r > 0.0, r, torch.ones_like(r))
    return torch.where(r > 0.0, off, math.sqrt(2.0 / math.pi) / torch.sqrt(s2))


def _orbitals(t, nocc, nvirt, g):
    """Overlap-like matrix S (the Gram matrix of Gaussians beside the atoms, so positive definite) and random
    S-orthonormal orbitals: as delocalised over the atoms as a flake's pi orbitals."""
    dev = t.pos.device
    ind = t.ind.long()
    shift = 0.45 * torch.randn((t.norb, 3), dtype=torch.float64, device=dev, generator=g)
    c = t.pos[ind] + shift
    d2 = torch.cdist(c, c, compute_mode="donot_use_mm_for_euclid_dist") ** 2
    S = 0.8 * torch.exp(-0.35 * d2)
    S.fill_diagonal_(1.0)
    L = torch.linalg.cholesky(S)
    Q, _ = torch.linalg.qr(torch.randn((t.norb, nocc + nvirt), dtype=torch.float64, device=dev, generator=g))
    C = torch.linalg.solve_triangular(L.mT, Q, upper=True)
    return S, C[:, :nocc].contiguous(), C[:, nocc:].contiguous()


def _pair_charges(t, C1, S1, C2, S2):
    """q^{pq}_A = 1/2 sum_{mu in A} (C1 S2 + S1 C2) in plain torch, one atom at a time."""
    out = torch.empty((t.nat, C1.shape[1], C2.shape[1]), dtype=torch.float64, device=C1.device)
    f = 0
    for A, n in enumerate(t.opa.tolist()):
        s = slice(f, f + n)
        torch.matmul(0.5 * torch.cat([C1[s], S1[s]]).T, torch.cat([S2[s], C2[s]]), out=out[A])
        f += n
    return out


def _energies(nocc, nvirt, dev, g):
    """omega_ia = e_a - e_i of a closed shell with a gap of about 2 eV (Hartree)."""
    eo = -0.24 - 0.55 * torch.sort(torch.rand(nocc, dtype=torch.float64, device=dev, generator=g), descending=True)[0]
    ev = -0.16 + 0.60 * torch.sort(torch.rand(nvirt, dtype=torch.float64, device=dev, generator=g))[0]
    return (ev[None, :] - eo[:, None]).contiguous()


def _product_inputs(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    t = _Tables(_molecule(case, seed), dev)
    no, nv, m = case["nocc"], case["nvirt"], case.get("m", 1)
    s = dict(op=case["op"], t=t, no=no, nv=nv, m=m)
    s["S"], s["Co"], s["Cv"] = _orbitals(t, no, nv, g)
    if case["op"] == "charges":
        return s
    r = _distances(t.pos)[0]
    s["gamma"], s["gamma_lr"] = _gamma(r, t.sigma, 0.0), _gamma(r, t.sigma, 0.5 * R_LR ** 2)
    s["omega"] = _energies(no, nv, dev, g)
    So, Sv = s["S"] @ s["Co"], s["S"] @ s["Cv"]
    s["q_ov"] = _pair_charges(t, s["Co"], So, s["Cv"], Sv)
    if case["op"] == "apbv":
        s["q_oo"] = _pair_charges(t, s["Co"], So, s["Co"], So)
        s["q_vv"] = _pair_charges(t, s["Cv"], Sv, s["Cv"], Sv)
    # expansion vectors: orthonormal columns with most weight on the lowest pairs
    V = torch.randn((no * nv, m), dtype=torch.float64, device=dev, generator=g)
    V /= (s["omega"].reshape(-1, 1) - 0.9 * s["omega"].min())
    s["V"] = torch.linalg.qr(V)[0].contiguous() if no * nv >= m else V
    ind = t.ind.long()
    s["G_lr"] = s["gamma_lr"][ind][:, ind].contiguous()
    return s


def prepare(case, seed):
    op = case["op"]
    native.load()
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    f64 = dict(dtype=torch.float64, device=dev)
    if op == "geometry":
        return dict(op=op, t=_Tables(_molecule(case, seed), dev))
    if op == "gradient":
        t = _Tables(_molecule(case, seed), dev)
        t.dircos = _distances(t.pos)
        t.mprox = _mprox(t.dircos[0])
        n = t.norb
        # adjoints fall off with the orbital distance like a density matrix
        decay = torch.exp(-0.15 * t.dircos[0])[t.ind.long()][:, t.ind.long()]
        adj = lambda: decay * torch.randn((n, n), generator=g, **f64)
        return dict(op=op, t=t, XS=adj(), XH=adj(), Yg=adj(), Ylr=adj() if case["lc"] else None)
    if op == "fp64gemm":
        # density- and overlap-like operands: rows of different magnitude
        scale = lambda k: torch.exp(torch.randn((k, 1), generator=g, **f64))
        A = scale(case["rows"]) * torch.randn((case["rows"], case["inner"]), generator=g, **f64)
        B = torch.randn((case["inner"], case["cols"]), generator=g, **f64) * scale(case["cols"]).T
        return dict(op=op, A=A, B=B, out=torch.empty((case["rows"], case["cols"]), **f64))
    if op == "train":
        n = case["samples"]
        net = learned.GuessNet(device=dev, seed=seed)
        feats = torch.randn((n, learned.NFEAT), device=dev, generator=g)
        feats = feats * torch.linspace(0.05, 3.0, learned.NFEAT, device=dev) + 0.4
        net.fit_statistics(feats)
        targets = 0.3 * torch.rand((n, learned.NOUT), device=dev, generator=g) ** 2
        weights = 0.25 + torch.rand(n, device=dev, generator=g)
        return dict(op=op, net=net, feats=feats, targets=targets, weights=weights)
    if op == "solve":
        return dict(op=op, mol=_molecule(case, seed), nstates=case["nstates"])
    s = _product_inputs(case, seed)
    t, L, m = s["t"], native.load(), s["m"]
    if op in ("exact_lc", "mixed_lc"):
        cls = lr_tddftb.ExchangeOzaki if op == "exact_lc" else lr_tddftb.ExchangeMixed
        s["product"] = cls(s["gamma"], s["G_lr"], s["q_ov"], s["omega"].reshape(-1), s["Co"], s["Cv"], s["S"], t.nat,
                           s["no"], s["nv"], native.Workspace(dev), lc=1)
        return s
    size = {"charges": lambda: L.dftb_trans_charges_workspace_size(t.norb, s["no"], s["nv"]),
            "hermitian": lambda: L.dftb_hermitian_rv_workspace_size(t.nat, m),
            "apbv": lambda: L.dftb_apbv_workspace_size(t.nat, s["no"], s["nv"], m)}[op]()
    s["work"] = native.Workspace(dev).get(size)
    return s


# ---------------------------------------------------------------- one pass
def _geometry_pass(t):
    P, st, dev = native.ptr, native.stream(), t.pos.device
    nat, n, p, tb = t.nat, t.norb, t.par, t.tables
    new = lambda *shape: torch.empty(shape, dtype=torch.float64, device=dev)
    r, x, y, z = new(nat, nat), new(nat, nat), new(nat, nat), new(nat, nat)
    native.call("dftb_directional_cosines", nat, P(t.pos), P(r), P(x), P(y), P(z), st)
    mp = _mprox(r)
    S, H0, D = new(n, n), new(n, n), new(3, n, n)
    native.call("dftb_h0_and_s", n, nat, P(t.ind), P(t.typ), P(t.ls), P(t.ms), P(r), P(x), P(y), P(z), P(mp),
                P(t.orben), p.deg, P(tb["tab_filled_SH0"]), P(tb["S_knots"]), P(tb["S_coefs"]), P(tb["H_knots"]),
                P(tb["H_coefs"]), p.npair, p.nsk, p.npts, P(S), P(H0), st)
    native.call("dftb_dipole_matrix", n, nat, P(t.ind), P(t.typ), P(t.ls), P(t.ms), P(r), P(x), P(y), P(z), P(t.pos),
                P(mp), P(S), p.deg, P(tb["tab_filled_D"]), P(tb["D_knots"]), P(tb["D_coefs"]), p.npair, p.nskd, p.npts,
                P(D), st)
    g, glr, G = new(nat, nat), new(nat, nat), new(n, n)
    native.call("dftb_gamma_matrices", nat, P(r), P(t.sigma), R_LR, P(g), P(glr), st)
    native.call("dftb_ao_expand", n, nat, P(t.ind), P(glr), P(G), st)
    return dict(r=r, x=x, y=y, z=z, S=S, H0=H0, D=D, g=g, glr=glr, G=G)


def run(s):
    op = s["op"]
    P, st = native.ptr, native.stream()
    if op == "geometry":
        return _geometry_pass(s["t"])
    if op == "gradient":
        t = s["t"]
        return gradients.contract(t, t.par, R_LR, s["XS"], s["XH"], s["Yg"], s["Ylr"], True)
    if op == "fp64gemm":
        return ozaki.matmul(s["A"], s["B"], out=s["out"])
    if op == "train":
        loss, grads = s["net"].loss_and_gradients(s["feats"], s["targets"], s["weights"])
        return dict(loss=loss, grads=grads)
    if op == "solve":
        td = lr_tddftb.LR_TDDFTB(s["mol"], long_range_correction=0)
        td.setGeometry(s["mol"])
        Omega, f = td.getEnergies(nstates=s["nstates"], diag_conv=1.0e-6, diag_maxiter=100)
        return dict(Omega=Omega, f=f, charges=td.dftb2.getPartialCharges(), levels=td.dftb2.getKSEnergies())
    t, no, nv, m = s["t"], s["no"], s["nv"], s["m"]
    if op in ("exact_lc", "mixed_lc"):
        return s["product"](s["V"])
    dev = t.pos.device
    new = lambda *shape: torch.empty(shape, dtype=torch.float64, device=dev)
    if op == "charges":
        oo, ov, vv = new(t.nat, no, no), new(t.nat, no, nv), new(t.nat, nv, nv)
        native.call("dftb_trans_charges", t.norb, t.nat, no, nv, P(s["Co"]), P(s["Cv"]), P(s["S"]), P(t.opa), P(oo),
                    P(ov), P(vv), P(s["work"]), s["work"].numel(), st)
        return oo, ov, vv
    if op == "hermitian":
        U = new(no * nv, m)
        native.call("dftb_hermitian_rv", t.nat, no, nv, m, P(s["gamma"]), P(s["q_ov"]), P(s["omega"]), P(s["V"]), P(U),
                    P(s["work"]), s["work"].numel(), st)
        return U
    plus, minus = new(no * nv, m), new(no * nv, m)
    for name, U in (("dftb_apbv", plus), ("dftb_ambv", minus)):
        native.call(name, t.nat, no, nv, m, 1, P(s["gamma"]), P(s["gamma_lr"]), P(s["q_oo"]), P(s["q_ov"]),
                    P(s["q_vv"]), P(s["omega"]), P(s["V"]), P(U), P(s["work"]), s["work"].numel(), st)
    return plus, minus


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    op = case["op"]
    if op == "train":
        n, H = case["samples"], learned.HIDDEN
        # forward: 64x256, 256x256, 256x2; backward: their weight gradients and two input gradients
        return dict(bytes=n * 4.0 * (8 + 2 + 1), flops=2.0 * n * (3 * 64 * H + 3 * H * H + 3 * 2 * H))
    if op == "fp64gemm":
        m, n, k = case["rows"], case["cols"], case["inner"]
        return dict(bytes=8.0 * (m * k + k * n + m * n), flops=2.0 * m * n * k)
    mol = _molecule(case, 0)
    nat = float(len(mol))
    n = float(_norb(case))
    if op == "solve":
        # about 26 SCC iterations of an eigensolve and its transforms, 12 Davidson iterations
        return dict(bytes=8.0 * (nat * n * n / 4 + 8 * n * n), flops=26 * 22.0 * n ** 3 + 12 * case["nstates"] * nat * n * n)
    if op == "geometry":
        return dict(bytes=8.0 * (6 * n * n + 6 * nat * nat), flops=60.0 * n * n)
    if op == "gradient":
        return dict(bytes=8.0 * ((4 if case["lc"] else 3) * n * n + 4 * nat * nat), flops=100.0 * n * n)
    no, nv = float(case["nocc"]), float(case["nvirt"])
    if op == "charges":
        pairs = no * no + no * nv + nv * nv
        return dict(bytes=8.0 * (nat * pairs + n * n + n * (no + nv)), flops=2.0 * n * n * (no + nv) + 4.0 * n * pairs)
    m = float(case["m"])
    if op == "hermitian":
        return dict(bytes=8.0 * (nat * no * nv + 2 * no * nv * m), flops=4.0 * nat * no * nv * m)
    if op == "apbv":
        per = nat * (no * no * nv + no * nv * nv)
        return dict(bytes=16.0 * (nat * (no * no + no * nv + nv * nv) + 2 * no * nv * m), flops=2 * m * (4.0 * per))
    # W, N, P1|P2, K1;K2 of every column and the two Coulomb products
    lc = 4.0 * n * no * nv + 8.0 * n * n * no + 16.0 * n * n * nv + 8.0 * n * no * nv
    return dict(bytes=8.0 * (nat * no * nv + 3 * no * nv * m + n * n), flops=m * (lc + 4.0 * nat * no * nv))


# ---------------------------------------------------------------- plain FP64 restatements
def _basis(t, l, x, degree):
    """The degree + 1 B-splines that live on knot interval l (1-based) at x (de Boor-Cox)."""
    h = [torch.ones_like(x)] + [torch.zeros_like(x) for _ in range(degree)]
    for j in range(1, degree + 1):
        prev = list(h)
        h[0] = torch.zeros_like(x)
        for i in range(1, j + 1):
            hi, lo = t[l + i - 1], t[l + i - j - 1]
            f = prev[i - 1] / (hi - lo)
            h[i - 1] = h[i - 1] + f * (hi - x)
            h[i] = f * (x - lo)
    return h


def _value(t, c, x):
    """Cubic spline value with the uniform-knot interval rule of splines.f90:25-92."""
    n = t.numel()
    tb, te = t[3], t[n - 4]
    l = ((x - t[0]) / (t[5] - t[4])).long() + 1
    l = torch.where(x <= tb, 4, torch.where(x >= te, n - 4, l))
    l = torch.where(l < 3, 4, l)
    arg = torch.clamp(x, tb, te)
    out = torch.zeros_like(x)
    for j, h in enumerate(_basis(t, l, arg, 3)):
        i = l - 4 + j
        out = out + torch.where(i >= 0, c[i.clamp_min(0)] * h, torch.zeros_like(h))
    return out


def _interval(t, x):
    return torch.searchsorted(t, x, right=True).clamp(4, t.numel() - 4)


def _derivative(t, c, x, clamp=True):
    """First derivative of the cubic spline (FITPACK splder)."""
    n = t.numel()
    if clamp:
        x = torch.clamp(x, t[3], t[n - 4])
    l = _interval(t, x)
    out = torch.zeros_like(x)
    for j, h in enumerate(_basis(t, l, x, 2)):
        i = l - 4 + j
        out = out + 3.0 * (c[i + 1] - c[i]) / (t[i + 4] - t[i + 1]) * h
    return out


def _pair_tables(knots, coefs, filled, ipair, r, fn):
    """fn of every table for every atom pair: (tables, nat, nat)."""
    out = torch.zeros((knots.shape[1],) + tuple(r.shape), dtype=torch.float64, device=r.device)
    for p in range(knots.shape[0]):
        mask = ipair == p
        if not bool(mask.any()):
            continue
        x = r[mask]
        for k in range(knots.shape[1]):
            if filled[p, k] == 1:
                out[k][mask] = fn(knots[p, k], coefs[p, k], x)
    return out


_AXIS = {-1: 1, 0: 2, 1: 0}


def _orientation(t, e):
    """Per ordered atom pair (i of orbital mu, j of orbital nu): whether the pair is read as (mu, nu), and the
    direction from the first to the second centre."""
    straight = t.atype[:, None] <= t.atype[None, :]
    d = -torch.stack(e)                                  # (3, i, j): (R_j - R_i) / r
    d = torch.where(straight[None], d, -d)
    # at zero distance the direction is +z whatever the order of the centres
    d[:2].diagonal(dim1=1, dim2=2).zero_()
    d[2].fill_diagonal_(1.0)
    return straight, d


def _sk_elements(t, e, rule):
    """rule(l1, m1, l2, m2, straight, direction) of every orbital pair from atom-pair matrices, as the planes
    that the rule returns; orbital kinds are few, so each kind pair is one block of atom pairs."""
    ind, ls, ms = t.ind.tolist(), t.ls.tolist(), t.ms.tolist()
    kinds = {}
    for mu in range(t.norb):
        kinds.setdefault((ls[mu], ms[mu]), []).append(mu)
    out = None
    straight, d = _orientation(t, e)
    for k1, rows in kinds.items():
        for k2, cols in kinds.items():
            ri = torch.tensor([ind[q] for q in rows], device=d.device)
            ci = torch.tensor([ind[q] for q in cols], device=d.device)
            pair = (ri[:, None], ci[None, :])
            vals = rule(k1, k2, straight, d, pair)
            if out is None:
                out = torch.zeros((len(vals), t.norb, t.norb), dtype=torch.float64, device=d.device)
            for q, v in enumerate(vals):
                out[q][torch.tensor(rows, device=d.device)[:, None], torch.tensor(cols, device=d.device)[None, :]] = v
    return out


def _rule_value(T, k1, k2, straight, d, pair):
    """Slater-Koster value between kinds k1 (of mu) and k2 (of nu); the first centre is mu's where straight."""
    def one(a, b):
        (l1, m1), (l2, m2) = a, b
        e = [d[c][pair] for c in range(3)]
        if l1 == 0 and l2 == 0:
            return T[0][pair]
        if l1 == 0:
            return e[_AXIS[m2]] * T[2][pair]
        if l2 == 0:
            return e[_AXIS[m1]] * T[4][pair]
        p, q = _AXIS[m1], _AXIS[m2]
        v = e[p] * e[q] * (T[6][pair] - T[5][pair])
        return v + T[5][pair] if p == q else v
    return torch.where(straight[pair], one(k1, k2), one(k2, k1))


def _exact_geometry(case, seed):
    s = prepare(case, seed)
    t = s["t"]
    p, tb = t.par, t.tables
    r, x, y, z = _distances(t.pos)
    tmin, tmax = torch.minimum(t.atype[:, None], t.atype[None, :]), torch.maximum(t.atype[:, None], t.atype[None, :])
    ipair = (tmax * (tmax + 1) // 2 + tmin).long()
    prox = _mprox(r)
    TS = _pair_tables(tb["S_knots"], tb["S_coefs"], p.tab_filled_SH0, ipair, r, _value)
    TH = _pair_tables(tb["H_knots"], tb["H_coefs"], p.tab_filled_SH0, ipair, r, _value)
    TD = _pair_tables(tb["D_knots"], tb["D_coefs"], p.tab_filled_D, ipair, r, _value)
    e = (x, y, z)
    SH = _sk_elements(t, e, lambda k1, k2, st, d, pr: (_rule_value(TS, k1, k2, st, d, pr),
                                                       _rule_value(TH, k1, k2, st, d, pr)))
    ind = t.ind.long()
    same = ind[:, None] == ind[None, :]
    far = prox[ind][:, ind] == 0
    S = torch.where(same, torch.eye(t.norb, dtype=torch.float64, device=r.device), SH[0])
    H0 = torch.where(same, torch.diag(t.orben), SH[1])
    S[far], H0[far] = 0.0, 0.0
    lower = lambda M: torch.tril(M) + torch.tril(M, -1).T   # both triangles hold the lower one's element
    S, H0 = lower(S), lower(H0)

    def dipole(k1, k2, straight, d, pair):
        def one(a, b):
            (l1, m1), (l2, m2) = a, b
            e = [d[c][pair] for c in range(3)]
            if l1 == 0 and l2 == 0:
                return [e[c] * TD[3][pair] for c in range(3)]
            if l1 + l2 == 1:
                q = _AXIS[m2 if l1 == 0 else m1]
                pi, sg = (TD[1][pair], TD[4][pair]) if l1 == 0 else (TD[6][pair], TD[13][pair])
                return [(pi if c == q else 0.0) + e[c] * e[q] * (sg - pi) for c in range(3)]
            u, v = _AXIS[m1], _AXIS[m2]
            d7, d8, d14 = TD[7][pair], TD[8][pair], TD[14][pair]
            res = []
            for c in range(3):
                w = e[u] * e[c] * e[v] * (d14 - d7 - 2.0 * d8)
                w = w + (e[v] * d7 if u == c else 0.0) + (e[u] * d8 if c == v else 0.0) + (e[c] * d8 if u == v else 0.0)
                res.append(w)
            return res
        return [torch.where(straight[pair], a, b) for a, b in zip(one(k1, k2), one(k2, k1))]

    D = _sk_elements(t, e, dipole)
    straight = t.atype[:, None] <= t.atype[None, :]
    origin = torch.where(straight[None], t.pos.T[:, None, :].expand(3, t.nat, t.nat),
                         t.pos.T[:, :, None].expand(3, t.nat, t.nat))
    D = D + origin[:, ind][:, :, ind] * S[None]
    D[:, far] = 0.0
    D = torch.stack([lower(D[c]) for c in range(3)])
    g, glr = _gamma(r, t.sigma, 0.0), _gamma(r, t.sigma, 0.5 * R_LR ** 2)
    return dict(r=r, x=x, y=y, z=z, S=S, H0=H0, D=D, g=g, glr=glr, G=glr[ind][:, ind].contiguous())


def _exact_gradient(case, seed):
    s = prepare(case, seed)
    t = s["t"]
    p, tb = t.par, t.tables
    r, x, y, z = t.dircos
    e = (x, y, z)
    tmin, tmax = torch.minimum(t.atype[:, None], t.atype[None, :]), torch.maximum(t.atype[:, None], t.atype[None, :])
    ipair = (tmax * (tmax + 1) // 2 + tmin).long()
    ind = t.ind.long()
    near = (ind[:, None] != ind[None, :]) & (t.mprox[ind][:, ind] != 0)
    safe = torch.where(r > 0.0, r, torch.ones_like(r))
    grad = torch.zeros((t.nat, 3), dtype=torch.float64, device=r.device)
    for X, kn, co in ((s["XS"], "S_knots", "S_coefs"), (s["XH"], "H_knots", "H_coefs")):
        T = _pair_tables(tb[kn], tb[co], p.tab_filled_SH0, ipair, r, _value)
        dT = _pair_tables(tb[kn], tb[co], p.tab_filled_SH0, ipair, r, _derivative)

        def rule(k1, k2, straight, d, pair, T=T, dT=dT):
            rr = safe[pair]

            def one(a, b):
                (l1, m1), (l2, m2) = a, b
                e = [d[c][pair] for c in range(3)]
                if l1 == 0 and l2 == 0:
                    return [dT[0][pair] * e[k] for k in range(3)]
                if l1 + l2 == 1:
                    q, tab = (_AXIS[m2], 2) if l1 == 0 else (_AXIS[m1], 4)
                    return [T[tab][pair] * ((1.0 if q == k else 0.0) - e[q] * e[k]) / rr + e[q] * dT[tab][pair] * e[k]
                            for k in range(3)]
                u, v = _AXIS[m1], _AXIS[m2]
                radial = e[u] * e[v] * (dT[6][pair] - dT[5][pair]) + (dT[5][pair] if u == v else 0.0)
                res = []
                for k in range(3):
                    ang = (e[v] if u == k else 0.0) + (e[u] if v == k else 0.0) - 2.0 * e[u] * e[v] * e[k]
                    res.append((T[6][pair] - T[5][pair]) * ang / rr + radial * e[k])
                return res
            # derivative with respect to the position of nu's atom
            return [torch.where(straight[pair], a, -b) for a, b in zip(one(k1, k2), one(k2, k1))]

        dM = _sk_elements(t, e, rule)
        W = torch.where(near, X + X.T, torch.zeros_like(X))
        for c in range(3):
            grad[:, c].index_add_(0, ind, (dM[c] * W).sum(0))
    blocks = lambda Y: torch.zeros((t.nat, t.nat), dtype=torch.float64, device=r.device).index_put_(
        (ind[:, None].expand(t.norb, t.norb), ind[None, :].expand(t.norb, t.norb)), Y + Y.T, accumulate=True)
    s2 = t.sigma[:, None] ** 2 + t.sigma[None, :] ** 2
    w = torch.zeros_like(r)
    for Y, extra in ((s["Yg"], 0.0), (s["Ylr"], 0.5 * R_LR ** 2)):
        if Y is not None:
            C = 1.0 / torch.sqrt(2.0 * (s2 + extra))
            w = w + (2.0 * C / math.sqrt(math.pi) * torch.exp(-(C * r) ** 2) / safe - torch.erf(C * r) / safe ** 2) * blocks(Y)
    for q in range(p.npair):
        dv = _derivative(tb["vrep_knots"][q], tb["vrep_coefs"][q], r, clamp=False)
        w = w + torch.where((ipair == q) & (r < tb["vrep_dmax"][q]), dv, torch.zeros_like(dv))
    w.fill_diagonal_(0.0)
    for c in range(3):
        grad[:, c] += (w * e[c]).sum(1)
    return grad.reshape(-1)


def _exact_exchange(s):
    """K1.V and K2.V in the AO-factorised form, one column at a time."""
    So, Sv = s["S"] @ s["Co"], s["S"] @ s["Cv"]
    Xo, Xb = torch.cat([s["Co"], So]), torch.cat([So, s["Co"]])
    Yv, Yb = torch.cat([s["Cv"], Sv]), torch.cat([Sv, s["Cv"]])
    n = s["S"].shape[0]
    K1, K2 = torch.empty_like(s["V"]), torch.empty_like(s["V"])
    for c in range(s["m"]):
        v = s["V"][:, c].reshape(s["no"], s["nv"])
        N = (Xo @ (v @ Yv.T)).view(2, n, 2, n) * s["G_lr"][None, :, None, :]
        N = N.reshape(2 * n, 2 * n)
        K1[:, c] = 0.25 * (Xb.T @ (N @ Yb)).reshape(-1)
        K2[:, c] = 0.25 * (Xb.T @ (N.T @ Yb)).reshape(-1)
    return K1, K2


def exact(case, seed):
    op = case["op"]
    if op == "solve":
        return None
    if op == "geometry":
        return _exact_geometry(case, seed)
    if op == "gradient":
        return _exact_gradient(case, seed)
    s = prepare(case, seed)
    if op == "fp64gemm":
        return s["A"] @ s["B"]
    if op == "train":
        net = s["net"]
        d = lambda v: v.double()
        X = (d(s["feats"]) - d(net.mean)) / d(net.std)
        W1 = d(net.W1)[:, :learned.NFEAT]
        Z1 = X @ W1.T + d(net.b1)
        H1 = Z1.clamp_min(0.0)
        Z2 = H1 @ d(net.W2).T + d(net.b2)
        H2 = Z2.clamp_min(0.0)
        Y = H2 @ d(net.W3).T + d(net.b3)
        diff = Y - d(s["targets"]) * d(net.target_scale)
        w = d(s["weights"])[:, None] / d(s["weights"]).sum()
        dY = 2.0 * w * diff
        dZ2 = (dY @ d(net.W3)) * (Z2 > 0.0)
        dZ1 = (dZ2 @ d(net.W2)) * (Z1 > 0.0)
        dW1 = torch.zeros((learned.HIDDEN, learned.FPAD), dtype=torch.float64, device=X.device)
        dW1[:, :learned.NFEAT] = dZ1.T @ X
        return dict(loss=float((w * diff * diff).sum()), grads=[dW1, dZ1.sum(0), dZ2.T @ H1, dZ2.sum(0), dY.T @ H2,
                                                                dY.sum(0)])
    t, V = s["t"], s.get("V")
    if op == "charges":
        Co, Cv = s["Co"], s["Cv"]
        So, Sv = s["S"] @ Co, s["S"] @ Cv
        return (_pair_charges(t, Co, So, Co, So), _pair_charges(t, Co, So, Cv, Sv), _pair_charges(t, Cv, Sv, Cv, Sv))
    om = s["omega"].reshape(-1, 1)
    q = s["q_ov"].reshape(t.nat, -1)
    if op == "hermitian":
        sq = torch.sqrt(om)
        return om * om * V + 4.0 * sq * (q.T @ (s["gamma"] @ (q @ (sq * V))))
    coul = om * V + 4.0 * (q.T @ (s["gamma"] @ (q @ V)))
    if op in ("exact_lc", "mixed_lc"):
        K1, K2 = _exact_exchange(s)
        return coul - K1 - K2, om * V + K2 - K1
    no, nv, m = s["no"], s["nv"], s["m"]
    v = V.reshape(no, nv, m)
    Z = torch.einsum("AB,Aij->Bij", s["gamma_lr"], s["q_oo"])
    Z2 = torch.einsum("AB,Bja->Aja", s["gamma_lr"], s["q_ov"])
    K1, K2 = torch.zeros_like(v), torch.zeros_like(v)
    for A in range(t.nat):
        T = torch.tensordot(Z[A], v, dims=([1], [0]))                         # (i, b, c)
        K1 += torch.einsum("ibc,ab->iac", T, s["q_vv"][A])
        W = torch.tensordot(Z2[A], v, dims=([0], [0]))                        # (a, b, c)
        K2 += torch.einsum("ib,abc->iac", s["q_ov"][A], W)
    K1, K2 = K1.reshape(no * nv, m), K2.reshape(no * nv, m)
    return coul - K1 - K2, om * V + K2 - K1
