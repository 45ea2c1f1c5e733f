"""Performance cases of dft_b200: the operators and whole solves that a user's program calls,
through the public Python face (`dft_b200.Engine`), over the sizes they are used at.

listed()           the fixed cases
draw(rng)          one more case of the same ranges
prepare(case, s)   inputs on the GPU, made from the seed
run(state)         one pass, returning everything the pass computes
work(case)         bytes and FP64 operations one pass cannot do without
exact(case, s)     the same outputs in plain 64-bit torch, where that is quick

Every field is FP64, x fastest, one array per field and band-major blocks, as the engine takes them.
"""
import math

import numpy as np
import torch

import dft_b200

DEV = "cuda"
F64 = torch.float64

# ----------------------------------------------------------------------- the cases ------


def listed():
    return [
        # one H psi block of the smallest benchmark molecule (H2, 48^3, 1 occupied + 3 extra bands):
        # a few microseconds, so the call itself counts
        {"name": "hpsi_48_b4", "op": "hpsi", "nx": 48, "ny": 48, "nz": 48, "bands": 4},
        # H psi on the cluster grid with a 16-band block: HBM-bound
        {"name": "hpsi_192_b16", "op": "hpsi", "nx": 192, "ny": 192, "nz": 192, "bands": 16},
        # the reference's own Poisson solve (Jacobi sweeps from zero to its stop rule) at H2's grid
        {"name": "hartree_jacobi_48", "op": "hartree", "nx": 48, "ny": 48, "nz": 48},
        # the fast Poisson solve (coarse start, multigrid cycles, Jacobi stop rule) on the H2O grid
        {"name": "poisson_multigrid_128", "op": "poisson", "nx": 128, "ny": 128, "nz": 128},
        # spin-polarised PBE potential and energy on the H2O grid
        {"name": "xc_pbe96_128", "op": "xc", "functional": "PBE96", "nx": 128, "ny": 128, "nz": 128},
        # LSDA on a ragged box
        {"name": "xc_pz81_ragged", "op": "xc", "functional": "PZ81", "nx": 75, "ny": 63, "nz": 91},
        # Gram product of the block eigensolver: a full basis of three 69-band blocks (the 20-atom
        # cluster) against its newest block, in FP64
        {"name": "gram_fp64_96", "op": "gram", "precision": 0, "nx": 96, "ny": 96, "nz": 96, "ka": 207, "kb": 69},
        # the same product of a mixed-precision solve (TF32 hi + lo on the tensor cores), ragged box
        {"name": "gram_tc_ragged", "op": "gram", "precision": 1, "nx": 112, "ny": 97, "nz": 101, "ka": 138,
         "kb": 69},
        # Ritz rotation of that basis
        {"name": "rotate_fp64_96", "op": "rotate", "precision": 0, "nx": 96, "ny": 96, "nz": 96, "ka": 138,
         "kb": 69},
        # one eigensolve of an H2O-sized molecule: 5 occupied + 7 extra bands from the seed vectors
        {"name": "eigensolve_64", "op": "eig", "nx": 64, "ny": 64, "nz": 64, "nocc": 5, "extra": 7},
        # a whole molecular SCF: H2 on 48^3 in the benchmark's fast configuration
        {"name": "scf_h2_48", "op": "scf", "functional": "PZ81", "n": 48},
        # the radial atoms Z = 1..30 with both functionals, all in one batch
        {"name": "atoms_60", "op": "atoms", "count": 60, "points": 2000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axes(rng, lo, hi, most):
    """Three axes of a box, odd and ragged ones among them, at most `most` points."""
    base = _log_int(rng, lo, hi)
    ax = [max(lo, min(hi, int(round(base * rng.uniform(0.85, 1.15))))) for _ in range(3)]
    while ax[0] * ax[1] * ax[2] > most:
        ax = [max(lo, a - 3) for a in ax]
    return {"nx": ax[0], "ny": ax[1], "nz": ax[2]}


def draw(rng):
    op = rng.choice(["hpsi", "hartree", "poisson", "xc", "gram", "rotate", "eig", "scf", "atoms"])
    if op == "hpsi":
        a = _axes(rng, 24, 192, 192 ** 3)
        return {"op": op, **a, "bands": _log_int(rng, 1, 16)}
    if op == "hartree":
        return {"op": op, **_axes(rng, 16, 64, 60 ** 3)}
    if op == "poisson":
        return {"op": op, **_axes(rng, 32, 128, 128 ** 3)}
    if op == "xc":
        return {"op": op, "functional": rng.choice(["PBE96", "PZ81"]), **_axes(rng, 24, 128, 128 ** 3)}
    if op in ("gram", "rotate"):
        kb = _log_int(rng, 2, 69)
        ka = max(kb, min(207, int(round(kb * rng.uniform(1.0, 3.0)))))
        return {"op": op, "precision": rng.choice([0, 1]), **_axes(rng, 32, 96, 96 ** 3), "ka": ka, "kb": kb}
    if op == "eig":
        return {"op": op, **_axes(rng, 28, 64, 64 ** 3), "nocc": rng.randint(1, 6), "extra": rng.randint(3, 7)}
    if op == "scf":
        return {"op": op, "functional": rng.choice(["PZ81", "PBE96"]), "n": rng.randint(36, 48)}
    return {"op": op, "count": _log_int(rng, 2, 60), "points": rng.randint(1200, 2000)}


# ----------------------------------------------------------------------- inputs ---------
H = 0.25  # grid spacing (bohr) of the operator cases


def _grid(case):
    n = (case["nx"], case["ny"], case["nz"])
    b = []
    for m in n:
        half = 0.5 * H * (m - 1)
        b += [-half, half]
    return dft_b200.CartesianGrid(*n, *b)


def _coords(grid):
    """x, y, z broadcast over (nz, ny, nx)."""
    b, n = grid.bounds, grid.shape
    ax = [b[2 * d] + torch.arange(n[d], dtype=F64, device=DEV) * ((b[2 * d + 1] - b[2 * d]) / (n[d] - 1))
          for d in range(3)]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _nuclei(rng, grid, count, zmax=8):
    """Random nuclei in the inner half of the box: (Z, x, y, z)."""
    b = grid.bounds
    out = []
    for _ in range(count):
        p = [0.5 * (b[2 * d] + b[2 * d + 1]) + 0.25 * (b[2 * d + 1] - b[2 * d]) * rng.uniform(-1, 1) for d in range(3)]
        out.append((int(rng.integers(1, zmax + 1)), *p))
    return out


def _r2(grid, c):
    x, y, z = _coords(grid)
    return (x - c[1]) ** 2 + (y - c[2]) ** 2 + (z - c[3]) ** 2


def _potential(grid, nuclei):
    """Screened nuclear wells, a molecule's effective potential without its grid-scale spikes."""
    v = torch.zeros((grid.nz, grid.ny, grid.nx), dtype=F64, device=DEV)
    for c in nuclei:
        r = torch.sqrt(_r2(grid, c) + 0.2)
        v -= c[0] * torch.exp(-0.4 * r) / r
    return v.reshape(-1)


def _density(grid, nuclei, scale=1.0, zeta=1.0):
    """Atomic densities with exponential tails, as SCF densities have."""
    n = torch.zeros((grid.nz, grid.ny, grid.nx), dtype=F64, device=DEV)
    for c in nuclei:
        z = zeta * (0.8 + 0.12 * c[0])
        n += scale * c[0] * z ** 3 / math.pi * torch.exp(-2.0 * z * torch.sqrt(_r2(grid, c) + 0.05))
    return n.reshape(-1)


def _bands(grid, nb, gen):
    """A band block: localised polynomials with some grid-scale content, normalised with dV."""
    x, y, z = _coords(grid)
    b = grid.bounds
    size = 0.5 * (b[1] - b[0])
    out = torch.empty((nb, grid.getSize()), dtype=F64, device=DEV)
    par = torch.rand((nb, 8), dtype=F64, device=DEV, generator=gen).cpu().numpy()
    dV = grid.getDx() * grid.getDy() * grid.getDz()
    for i in range(nb):
        p = par[i]
        c = [(2 * p[d] - 1) * 0.4 * size for d in range(3)]
        w = (0.15 + 0.4 * p[3]) * size
        f = torch.exp(-((x - c[0]) ** 2) / (2 * w * w)) * torch.exp(-((y - c[1]) ** 2) / (2 * w * w))
        f = f * torch.exp(-((z - c[2]) ** 2) / (2 * w * w))
        f = f * (p[4] - 0.5 + (p[5] - 0.5) * x + (p[6] - 0.5) * y + (p[7] - 0.5) * z)
        f = f.reshape(-1)
        f = f + 1e-3 * f.abs().max() * torch.randn(f.shape, dtype=F64, device=DEV, generator=gen)
        out[i] = f / math.sqrt(float((f * f).sum()) * dV)
    return out


def _h2(seed, n):
    """H2 near its bond length, turned and shifted at random, no nucleus at a node."""
    rng = np.random.default_rng(seed)
    h = 0.3
    half = round(0.5 * h * (n - 1), 10)
    while True:
        u = rng.standard_normal(3)
        u /= np.linalg.norm(u)
        c = rng.uniform(-0.15, 0.15, 3)
        d = 0.5 * rng.uniform(1.3, 1.5)
        pts = [c + d * u, c - d * u]
        off = [np.linalg.norm(((p + half) / h - np.round((p + half) / h)) * h) for p in pts]
        if min(off) > 0.08:
            break
    m = dft_b200.Molecule(0)
    for p in pts:
        m.addNucleus(1, *map(float, p))
    return dft_b200.CartesianGrid(n, n, n, -half, half, -half, half, -half, half), m


def prepare(case, seed):
    eng = dft_b200.engine()  # one engine per program
    op = case["op"]
    rng = np.random.default_rng(seed)
    if op == "scf":
        grid, mol = _h2(seed, case["n"])
        # the fast configuration: multigrid Poisson starts, started from the mixer's combination,
        # Pulay mixing, atoms start, eigensolver tolerance that follows the density
        o = dft_b200.default_scf_options(
            stop_abs_de=1e-7, stop_abs_deig=1e-7, stop_abs_drho=5e-7, extra_bands=3, max_iterations=60,
            poisson_start=dft_b200.POISSON_MULTIGRID, eig_mixed_precision=1, eig_preconditioner=-2, mixer=1,
            adaptive_eig_tol=1, poisson_predict=1, initial_density=1, eig_tol=1e-9)
        return {"op": op, "eng": eng, "grid": grid, "mol": mol, "functional": case["functional"], "options": o}
    if op == "atoms":
        # the radial table of the elements: heavy ones always in it, the box radius is the user's
        n = case["count"]
        Z = [30 - (i // 2) % 30 for i in range(n)]
        kinds = [("PZ81", "PBE96")[i % 2] for i in range(n)]
        return {"op": op, "eng": eng, "Z": Z, "kinds": kinds, "points": case["points"],
                "rmax": float(rng.uniform(28.0, 32.0)) * case["points"] / 2000.0}
    grid = _grid(case)
    N = grid.getSize()
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    s = {"op": op, "eng": eng, "grid": grid, "N": N}

    def new(n):
        return torch.empty(n, dtype=F64, device=DEV)

    if op == "hpsi":
        s["V"] = _potential(grid, _nuclei(rng, grid, 4))
        s["psi"] = _bands(grid, case["bands"], gen)
        s["out"] = torch.empty_like(s["psi"])
    elif op in ("hartree", "poisson"):
        s["rho"] = _density(grid, _nuclei(rng, grid, 3), zeta=0.6)
        s["vh"] = new(N)
    elif op == "xc":
        nuc = _nuclei(rng, grid, 3)
        s["functional"] = case["functional"]
        s["na"], s["nb"] = _density(grid, nuc, 0.55, 0.9), _density(grid, nuc[:2], 0.45, 0.8)
        s["va"], s["vb"] = new(N), new(N)
    elif op == "gram":
        s["A"], s["B"], s["precision"] = _bands(grid, case["ka"], gen), _bands(grid, case["kb"], gen), case["precision"]
    elif op == "rotate":
        s["A"], s["precision"] = _bands(grid, case["ka"], gen), case["precision"]
        q, _ = np.linalg.qr(rng.standard_normal((case["ka"], case["kb"])))
        s["Y"] = np.ascontiguousarray(q)
        s["out"] = torch.empty((case["kb"], N), dtype=F64, device=DEV)
    else:  # eig
        s["V"] = _potential(grid, _nuclei(rng, grid, 3))
        s["nocc"], s["nb"] = case["nocc"], case["nocc"] + case["extra"]
        s["psi"] = torch.empty((s["nb"], N), dtype=F64, device=DEV)
    return s


# ----------------------------------------------------------------------- one pass -------
def run(s):
    eng, op = s["eng"], s["op"]
    if op == "hpsi":
        eng.apply_hamiltonian(s["grid"], s["V"], s["psi"], s["out"], s["psi"].shape[0], s["N"])
        return s["out"]
    if op == "hartree":
        sweeps, last = eng.hartree(s["grid"], s["rho"], s["vh"])
        return {"v": s["vh"], "sweeps": sweeps, "last": last}
    if op == "poisson":
        eng.poisson_start(s["grid"], None, s["rho"], s["vh"], multigrid_cycles=40)
        eng.hartree_from_guess(s["grid"], s["rho"], s["vh"])
        return s["vh"]
    if op == "xc":
        e = eng.xc(s["grid"], s["functional"], s["na"], s["nb"], s["va"], s["vb"], energy=True)
        return {"va": s["va"], "vb": s["vb"], "energy": e}
    if op == "gram":
        return eng.gram(s["grid"], s["A"], s["N"], s["A"].shape[0], s["B"], s["N"], s["B"].shape[0],
                        precision=s["precision"])
    if op == "rotate":
        eng.rotate(s["grid"], s["A"], s["N"], s["A"].shape[0], s["Y"], s["out"], s["N"], precision=s["precision"])
        return s["out"]
    if op == "eig":
        e, _ = eng.solve_orbitals(s["grid"], s["V"], s["nocc"], s["nb"], s["psi"], s["N"], preconditioner=-2)
        # the extra bands only stay ahead of the occupied ones: they are not converged
        return {"eigenvalues": e[: s["nocc"]], "orbitals": s["psi"][: s["nocc"]]}
    if op == "scf":
        r = eng.scf_molecule(s["grid"], s["mol"], 0, 1, s["functional"], s["options"], want_density=True)
        e = r.energy
        return {"energy": np.array([e.kinetic, e.external, e.hartree, e.exchangeCorrelation, e.nuclearRepulsion,
                                    e.total]),
                "eigenvalues": np.array(r.eigenvalues), "alpha": r.alphaDensity, "beta": r.betaDensity}
    rs = eng.solve_atoms(s["Z"], s["kinds"], s["points"], s["rmax"])
    lv = np.zeros((len(rs), 16))
    for i, r in enumerate(rs):
        lv[i, : len(r.eigenvalues)] = r.eigenvalues
    # (the final density difference and residual are rounding noise below the stop: not compared)
    return {"energy": np.array([[r.energy.kinetic, r.energy.external, r.energy.hartree, r.energy.exchangeCorrelation,
                                 r.energy.total] for r in rs]), "eigenvalues": lv,
            "iterations": np.array([r.iterations for r in rs]), "status": np.array([r.status for r in rs]),
            "converged": np.array([int(r.converged) for r in rs])}


# ----------------------------------------------------------------------- work -----------
def work(case):
    op = case["op"]
    if op == "scf":
        # one read of the nuclei's potential, one write of each spin density
        N = case["n"] ** 3
        return {"bytes": 8.0 * 3 * N, "flops": 60.0 * N}
    if op == "atoms":
        # per run: the grid's potential, two densities and the orbitals once
        return {"bytes": 8.0 * 10 * case["points"] * case["count"], "flops": 200.0 * case["points"] * case["count"]}
    N = case["nx"] * case["ny"] * case["nz"]
    if op == "hpsi":
        return {"bytes": 8.0 * N * (2 * case["bands"] + 1), "flops": 15.0 * N * case["bands"]}
    if op in ("hartree", "poisson"):
        return {"bytes": 16.0 * N, "flops": 30.0 * N}
    if op == "xc":
        return {"bytes": 32.0 * N, "flops": (700.0 if case["functional"] == "PBE96" else 300.0) * N}
    if op == "gram":
        return {"bytes": 8.0 * N * (case["ka"] + case["kb"]), "flops": 2.0 * N * case["ka"] * case["kb"]}
    if op == "rotate":
        return {"bytes": 8.0 * N * (case["ka"] + case["kb"]), "flops": 2.0 * N * case["ka"] * case["kb"]}
    return {"bytes": 8.0 * N * (1 + case["nocc"] + case["extra"]), "flops": 100.0 * N * (case["nocc"] + case["extra"])}


# ----------------------------------------------------------------------- 64-bit values --
def exact(case, seed):
    op = case["op"]
    if op in ("scf", "atoms"):
        return None  # a whole SCF, or up to 60 of them point by point: minutes
    s = prepare(case, seed)
    g = s["grid"]
    dV = g.getDx() * g.getDy() * g.getDz()
    if op == "hpsi":
        return torch.stack([_apply_h(g, s["V"], p) for p in s["psi"]])
    if op == "hartree":
        return _jacobi(g, s["rho"])
    if op == "poisson":
        return _dirichlet(g, 4.0 * math.pi * s["rho"], 0.0)
    if op == "xc":
        return (_pbe if case["functional"] == "PBE96" else _pz)(g, s["na"], s["nb"], dV)
    if op == "gram":
        return (dV * (s["A"] @ s["B"].T)).cpu().numpy()
    if op == "rotate":
        return torch.from_numpy(s["Y"]).to(DEV).T @ s["A"]
    return {"eigenvalues": _lowest(g, s["V"], s["nocc"]), "orbitals": None}  # orbitals: up to a sign


def _apply_h(g, V, psi):
    p = psi.view(g.nz, g.ny, g.nx)
    lap = -2.0 * (1.0 / g.getDx() ** 2 + 1.0 / g.getDy() ** 2 + 1.0 / g.getDz() ** 2) * p
    for d, h in ((2, g.getDx()), (1, g.getDy()), (0, g.getDz())):
        n = p.shape[d]
        lap.narrow(d, 1, n - 1).add_(p.narrow(d, 0, n - 1), alpha=1.0 / (h * h))
        lap.narrow(d, 0, n - 1).add_(p.narrow(d, 1, n - 1), alpha=1.0 / (h * h))
    return (-0.5 * lap).reshape(-1) + V * psi


def _jacobi(g, rho, tol=1e-8, cap=10000):
    """Jacobi sweeps from zero with zero faces until max|dV| < tol."""
    w = [1.0 / g.getDx() ** 2, 1.0 / g.getDy() ** 2, 1.0 / g.getDz() ** 2]
    den = 2.0 * sum(w)
    v = torch.zeros((g.nz, g.ny, g.nx), dtype=F64, device=DEV)
    src = (4.0 * math.pi * rho).view(g.nz, g.ny, g.nx)[1:-1, 1:-1, 1:-1]
    d = torch.zeros((), dtype=F64, device=DEV)
    for sweep in range(1, cap + 1):
        c = v[1:-1, 1:-1, 1:-1]
        new = (w[0] * (v[1:-1, 1:-1, :-2] + v[1:-1, 1:-1, 2:]) + w[1] * (v[1:-1, :-2, 1:-1] + v[1:-1, 2:, 1:-1]) +
               w[2] * (v[:-2, 1:-1, 1:-1] + v[2:, 1:-1, 1:-1]) + src) / den
        d = (new - c).abs().max()
        u = torch.zeros_like(v)
        u[1:-1, 1:-1, 1:-1] = new
        v = u
        if float(d) < tol:
            break
    return {"v": v.reshape(-1), "sweeps": None, "last": float(d)}


def _sines(m):
    k = torch.arange(1, m + 1, dtype=F64, device=DEV)
    return torch.sin(math.pi / (m + 1) * torch.outer(k, k)) * math.sqrt(2.0 / (m + 1))


def _along(S, a):
    """The (symmetric) matrices S applied along the last three axes of a."""
    a = torch.einsum("ck,...ijk->...ijc", S[2], a)
    a = torch.einsum("bj,...ijk->...ibk", S[1], a)
    return torch.einsum("ai,...ijk->...ajk", S[0], a)


def _dirichlet(g, src, shift):
    """(-lap_h + shift) v = src on the interior, zero faces, by sine transforms."""
    f = src.view(g.nz, g.ny, g.nx)[1:-1, 1:-1, 1:-1]
    n, h = (g.nz - 2, g.ny - 2, g.nx - 2), (g.getDz(), g.getDy(), g.getDx())
    S = [_sines(m) for m in n]
    lam = [4.0 / (q * q) * torch.sin(0.5 * math.pi * torch.arange(1, m + 1, dtype=F64, device=DEV) / (m + 1)) ** 2
           for m, q in zip(n, h)]
    den = lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :] + shift

    def transform(a):
        return _along(S, a)

    v = torch.zeros((g.nz, g.ny, g.nx), dtype=F64, device=DEV)
    v[1:-1, 1:-1, 1:-1] = transform(transform(f) / den)
    return v.reshape(-1)


def _lowest(g, V, nocc, tol=1e-9, iterations=300):
    """The lowest eigenvalues of H by a preconditioned block method (sine-transform (T + 1)^-1)."""
    m, N = nocc + 6, g.getSize()
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1)
    n, h = (g.nz, g.ny, g.nx), (g.getDz(), g.getDy(), g.getDx())
    S = [_sines(q) for q in n]
    lam = [2.0 / (q * q) * torch.sin(0.5 * math.pi * torch.arange(1, k + 1, dtype=F64, device=DEV) / (k + 1)) ** 2
           for k, q in zip(n, h)]
    den = lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :] + 1.0

    def solve(r):
        return _along(S, _along(S, r.view(-1, *n)) / den).reshape(-1, N)

    r2 = torch.zeros(n, dtype=F64, device=DEV)
    for c in _coords(g):
        r2 = r2 + c * c
    X = torch.randn((m, N), dtype=F64, device=DEV, generator=gen) * torch.exp(-0.1 * r2).reshape(-1)
    X = solve(X)
    P = X[:0]
    for _ in range(iterations):
        Q, _ = torch.linalg.qr(X.T)
        X = Q.T
        HX = torch.stack([_apply_h(g, V, p) for p in X])
        th, U = torch.linalg.eigh(X @ HX.T)
        X, HX = U.T @ X, U.T @ HX
        R = HX - th[:, None] * X
        if float(R[:nocc].norm(dim=1).max()) < tol:
            break
        B, _ = torch.linalg.qr(torch.cat([X, solve(R), P]).T)
        B = B.T
        HB = torch.stack([_apply_h(g, V, p) for p in B])
        _, U = torch.linalg.eigh(B @ HB.T)
        Xn = U[:, :m].T @ B
        P = Xn - (Xn @ X.T) @ X
        X = Xn
    return th[:nocc].cpu().numpy()


def _diff(f, d, h):
    """Central difference along axis d, one-sided at the faces."""
    n = f.shape[d]
    out = torch.empty_like(f)
    out.narrow(d, 1, n - 2).copy_((f.narrow(d, 2, n - 2) - f.narrow(d, 0, n - 2)) / (2.0 * h))
    out.narrow(d, 0, 1).copy_((f.narrow(d, 1, 1) - f.narrow(d, 0, 1)) / h)
    out.narrow(d, n - 1, 1).copy_((f.narrow(d, n - 1, 1) - f.narrow(d, n - 2, 1)) / h)
    return out


def _pz(g, a, b, dV):
    """Slater exchange and Perdew-Zunger 1981 correlation; v = d(n eps)/dn_sigma."""
    n = a + b
    z = (a - b) / n
    rs = (3.0 / (4.0 * math.pi * n)) ** (1.0 / 3.0)

    def corr(A, B, C, D, gm, b1, b2):
        lo = rs < 1.0
        l, q = torch.log(rs), torch.sqrt(rs)
        den = 1.0 + b1 * q + b2 * rs
        e = torch.where(lo, A * l + B + C * rs * l + D * rs, gm / den)
        d = torch.where(lo, A / rs + C * (l + 1.0) + D, -gm * (b1 / (2.0 * q) + b2) / den ** 2)
        return e, d

    e0, d0 = corr(0.0311, -0.0480, 0.0020, -0.0116, -0.1423, 1.0529, 0.3334)
    e1, d1 = corr(0.01555, -0.0269, 0.0007, -0.0048, -0.0843, 1.3981, 0.2611)
    p43 = (1 + z) ** (4.0 / 3.0) + (1 - z) ** (4.0 / 3.0)
    p13 = (1 + z) ** (1.0 / 3.0) - (1 - z) ** (1.0 / 3.0)
    fd = 2.0 ** (4.0 / 3.0) - 2.0
    f, df = (p43 - 2.0) / fd, 4.0 / 3.0 * p13 / fd
    ex0 = -0.7385587663820223 * n ** (1.0 / 3.0)
    ex = ex0 * 0.5 * p43
    exc = ex + e0 + f * (e1 - e0)
    drs = -ex / rs + d0 + f * (d1 - d0)
    dz = ex0 * 2.0 / 3.0 * p13 + df * (e1 - e0)
    r = exc - rs * drs / 3.0
    on = n > 1e-20
    zero = torch.zeros_like(n)
    return {"va": torch.where(on, r + (1 - z) * dz, zero), "vb": torch.where(on, r - (1 + z) * dz, zero),
            "energy": float(torch.where(on, n * exc, zero).sum()) * dV}


def _pbe(g, a, b, dV):
    """PBE exchange (spin scaling) and correlation on PW92, the gradient terms by central
    differences of |grad n_sigma|; v = d(n eps)/dn_sigma - div(c_sigma grad n_sigma)."""
    shape = (g.nz, g.ny, g.nx)
    h = (g.getDx(), g.getDy(), g.getDz())
    A, B = a.view(shape), b.view(shape)
    ga3, gb3 = [[_diff(F, 2 - d, h[d]) for d in range(3)] for F in (A, B)]
    ga, gb = [torch.sqrt(q[0] ** 2 + q[1] ** 2 + q[2] ** 2) for q in (ga3, gb3)]
    n = A + B
    third = 1.0 / 3.0
    kappa, mu = 0.804, 0.2195149727645171
    gamma, beta = 0.031090690869654895, 0.06672455060314922
    delta, fg = beta / gamma, 0.51984209978974632953
    fzz, eta = 8.0 / (9.0 * fg), 1.0e-12

    def exchange(r, q):
        r13 = r ** third
        exu = -0.73855876638202240588 * r13
        s = q / (2.0 * 3.09366772628014 * r13 * r)
        p0 = 1.0 + mu / kappa * s * s
        fx = 1.0 + kappa - kappa / p0
        fs = 2.0 * mu / (p0 * p0)
        return (r * exu * fx, exu * 4.0 / 3.0 * (fx - s * s * fs),
                -0.73855876638202240588 * 0.161620459673995 * s * fs)

    def gcor(q, a1, b1, b2, b3, b4, x):
        q0 = -2.0 * q * (1.0 + a1 * x * x)
        q1 = 2.0 * q * x * (b1 + x * (b2 + x * (b3 + b4 * x)))
        l = torch.log(1.0 + 1.0 / q1)
        q3 = q * (b1 / x + 2.0 * b2 + x * (3.0 * b3 + 4.0 * b4 * x))
        return q0 * l, -2.0 * q * a1 * l - q0 * q3 / (q1 * (1.0 + q1))

    eda, dna, dga = exchange(2.0 * A, 2.0 * ga)
    edb, dnb, dgb = exchange(2.0 * B, 2.0 * gb)
    z = torch.clamp((A - B) / n, -1.0, 1.0)
    gm = ga + gb
    rs = (3.0 / (4.0 * math.pi * n)) ** third
    phi = 0.5 * ((1 + z) ** (2 * third) + (1 - z) ** (2 * third))
    ks = torch.sqrt(4.0 * (3.0 * math.pi ** 2 * n) ** third / math.pi)
    t = gm / (2.0 * ks * phi * n)
    x = torch.sqrt(rs)
    eu, eud = gcor(0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294, x)
    ep, epd = gcor(0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517, x)
    al, ad = gcor(0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671, x)
    z3, z4 = z ** 3, z ** 4
    f = ((1 + z) ** (4 * third) + (1 - z) ** (4 * third) - 2.0) / fg
    fz = 4.0 * third * ((1 + z) ** third - (1 - z) ** third) / fg
    ec = eu * (1.0 - f * z4) + ep * f * z4 - al * f * (1.0 - z4) / fzz
    ecrs = eud * (1.0 - f * z4) + epd * f * z4 - ad * f * (1.0 - z4) / fzz
    ecz = 4.0 * z3 * f * (ep - eu + al / fzz) + fz * (z4 * ep - z4 * eu - (1.0 - z4) * al / fzz)
    phi3 = phi ** 3
    arg = -ec / (gamma * phi3)
    bb = delta / torch.expm1(arg)
    t2 = t * t
    q4, q5 = 1.0 + bb * t2, 1.0 + bb * t2 + bb * bb * t2 * t2
    hh = phi3 * (beta / delta) * torch.log(1.0 + delta * q4 * t2 / q5)
    fac = delta / bb + 1.0
    bec = bb * bb * fac / (beta * phi3)
    q8 = q5 * q5 + delta * q4 * q5 * t2
    hb = -beta * phi3 * bb * t2 ** 3 * (2.0 + bb * t2) / q8
    hrs = -(rs / 3.0) * hb * bec * ecrs
    ht = 2.0 * beta * phi3 * (1.0 + 2.0 * bb * t2) / q8
    comm = hh + hrs - 7.0 * t2 * ht / 6.0
    gz = ((1 + z + eta) ** -third - (1 - z + eta) ** -third) / 3.0
    bg = -3.0 * bb * bb * ec * fac / (beta * phi3 * phi)
    hz = 3.0 * gz * hh / phi + hb * (bg * gz + bec * ecz)
    pref = hz - gz * t2 * ht / phi
    com = ec - rs * ecrs / 3.0 - z * ecz
    dgc = t * ht / (2.0 * ks * phi)
    on = n > 1e-20
    zero = torch.zeros_like(n)
    out = {}
    for name, d, c, g3 in (("va", dna + com + ecz + comm + pref * (1.0 - z), dga + dgc, ga3),
                           ("vb", dnb + com - ecz + comm - pref * (1.0 + z), dgb + dgc, gb3)):
        c = torch.where(on, c, zero)
        v = torch.where(on, d, zero)
        for q in range(3):
            v = v - _diff(c * g3[q], 2 - q, h[q])
        out[name] = torch.where(on, v, zero).reshape(-1)
    out["energy"] = float(torch.where(on, 0.5 * (eda + edb) + n * (ec + hh), zero).sum()) * dV
    return out
