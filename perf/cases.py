"""The work that a program using lynx_b200 has it do, for timing and for comparing results.

A case is one public call (or the few calls that belong together) of the CheFSI eigensolver path:
the Hamiltonian apply and its adjoint, the Chebyshev filter, a whole CheFSI pass with the density
of its orbitals, a batch of independent passes, the effective potential, and forces and stress.
The systems are silicon cells of 8, 64 and 216 atoms (grid spacing about 0.34 Bohr, 3 states per
atom or a little less, FD order 12, degree 20) and the two-atom FCC cell at k-points, with seeded
displaced atoms, a seeded potential and seeded orbitals.
"""
import math
import os
import tempfile

import numpy as np
import torch

from lynx_b200 import autograd, pseudo, solver
from lynx_b200 import cell as C
from lynx_b200.potential import EffectivePotential

DEV = "cuda:0" if torch.cuda.is_available() else "cpu"
BETA = 1000.0  # Fermi-Dirac smearing of 0.001 Ha


def listed():
    return [
        # one H psi of the smallest cell: what every operator call of a small system costs
        {"name": "apply_si8", "kind": "apply", "reps": 1, "shape": "30x30x30", "ncol": 24, "kpt": False},
        # differentiable H psi, forward and backward (gradients in the orbitals and the potential)
        {"name": "autograd_si64", "kind": "autograd", "reps": 2, "shape": "60x60x60", "ncol": 160},
        # the filter alone at an ordinary size, in the mixed path's precision
        {"name": "filter_si64_mixed", "kind": "filter", "reps": 2, "shape": "60x60x60", "ncol": 160, "kpt": False,
         "degree": 20, "precision": "mixed"},
        # ragged: odd grid, odd number of columns, another degree
        {"name": "filter_odd_mixed", "kind": "filter", "reps": 2, "shape": "51x57x63", "ncol": 97, "kpt": False,
         "degree": 16, "precision": "mixed"},
        # complex Bloch orbitals on the non-orthogonal primitive cell (one k-point of a k-grid)
        {"name": "filter_fcc_kpt_fp64", "kind": "filter", "reps": 0, "shape": "20x20x20", "ncol": 16, "kpt": True,
         "degree": 20, "precision": "fp64"},
        # eigensolver + density of one SCF iteration: the smallest cell, the ordinary one in both
        # precisions, the largest one
        {"name": "pass_si8_fp64", "kind": "pass", "reps": 1, "shape": "30x30x30", "ncol": 24, "precision": "fp64"},
        {"name": "pass_si64_fp64", "kind": "pass", "reps": 2, "shape": "60x60x60", "ncol": 160, "precision": "fp64"},
        {"name": "pass_si64_mixed", "kind": "pass", "reps": 2, "shape": "60x60x60", "ncol": 160, "precision": "mixed"},
        {"name": "pass_si216_mixed", "kind": "pass", "reps": 3, "shape": "90x90x90", "ncol": 520, "precision": "mixed"},
        # many small problems at once: the k-points of the FCC cell and an ensemble of strained Si8 cells
        {"name": "batch_kpt_ensemble", "kind": "batch", "kgrid": 3, "grid": 20, "ncol": 16, "cells": "24,26,28,30,32",
         "ncol_cell": 24, "precision": "mixed"},
        # the potential update of an SCF iteration at the largest grid
        {"name": "veff_si216", "kind": "veff", "reps": 3, "shape": "90x90x90"},
        # nonlocal forces, kinetic and nonlocal stress after convergence
        {"name": "forces_stress_si64", "kind": "forces", "reps": 2, "shape": "60x60x60", "ncol": 160, "kpt": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "filter", "filter", "filter", "pass", "pass", "pass", "autograd", "batch",
                       "veff", "forces"])
    if kind == "batch":
        return {"kind": "batch", "kgrid": rng.randint(1, 3), "grid": 2 * rng.randint(8, 12), "ncol": rng.randint(9, 20),
                "cells": ",".join(str(rng.randint(22, 32)) for _ in range(rng.randint(1, 6))), "ncol_cell": rng.randint(17, 30),
                "precision": rng.choice(["mixed", "fp64"])}
    kpt = kind in ("apply", "filter", "forces") and rng.random() < 0.35
    reps = rng.choice([0, 1]) if kpt else rng.choice([1, 2, 2, 3] if kind in ("pass", "veff", "filter") else [1, 2])
    per = (16, 24) if reps == 0 else (24, 32) if reps < 3 else (24, 30)
    n = max(1, reps)
    base = rng.randint(*per)  # the cells are cubic: the three counts lie close together
    shape = [max(per[0] * n, min(per[1] * n, n * base + rng.randint(-2, 2))) for _ in range(3)]
    if kind == "pass" and reps == 3:
        shape[0] -= shape[0] % 2
    case = {"kind": kind, "reps": reps, "shape": "x".join(map(str, shape))}
    if kind == "veff":
        return case
    top = {0: 24, 1: 40, 2: 200, 3: 520}[reps]
    if kind == "pass":  # enough states for the valence bands: 2 per atom and some empty ones
        nat = 8 * reps ** 3
        case["ncol"] = rng.randint(int(2.2 * nat), min(int(3.0 * nat), top))
        case["precision"] = "mixed" if reps == 3 else rng.choice(["mixed", "mixed", "fp64"])
        return case
    case["ncol"] = _log_int(rng, 1 if kind in ("apply", "filter") else 8, top)
    if kind in ("apply", "filter", "forces"):
        case["kpt"] = kpt
    if kind == "filter":
        case["degree"] = rng.randint(8, 24) if reps < 3 else rng.randint(8, 20)
        case["precision"] = "mixed" if reps == 3 else rng.choice(["mixed", "mixed", "fp64"])
    return case


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
_PSP = None


def _psp():
    global _PSP
    if _PSP is None:
        with tempfile.TemporaryDirectory() as d:
            _PSP = pseudo.read_psp8(pseudo.synthetic_si_psp8(os.path.join(d, "si.psp8")))
    return _PSP


def _shape(case):
    return tuple(int(n) for n in case["shape"].split("x"))


def _cells(case):
    return [int(n) for n in case["cells"].split(",")]


def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _gaussians(cl, pos, width):
    """Sum over atoms of exp(-r^2 / 2 width^2), periodic, on the grid (orthogonal cells)."""
    g = []
    for d in range(3):
        n, L = cl.shape[d], cl.lengths[d]
        x = torch.arange(n, device=DEV, dtype=torch.float64) * (L / n)
        p = torch.tensor(pos[:, d], device=DEV, dtype=torch.float64)
        r = x[None, :, None] - p[:, None, None] - L * torch.arange(-2, 3, device=DEV, dtype=torch.float64)
        g.append(torch.exp(-r * r / (2 * width * width)).sum(2))
    zy = (g[2][:, :, None] * g[1][:, None, :]).reshape(len(pos), -1)
    return (zy.T @ g[0]).reshape(-1)


def _system(case, seed, strain=None):
    """Cell, atoms, projector tables and potential: reps^3 conventional cells, or (reps 0) the FCC cell."""
    shape = _shape(case)
    if case["reps"] == 0:
        cl, pos = C.fcc_si_primitive(shape[0])
        cl.shape = shape
        pos = pos + np.random.default_rng(seed).normal(0.0, 0.02, pos.shape)
        pos = np.mod(pos, cl.lengths)
        V = torch.from_numpy(C.synthetic_veff(cl, pos)).to(DEV)
    else:
        cl, pos = C.diamond_si(case["reps"], shape, displace=0.02, strain=strain, seed=seed)
        V = -1.2 * _gaussians(cl, pos, 1.1)
    V = V + 1e-3 * torch.randn(V.shape, device=DEV, dtype=torch.float64, generator=_rng(seed))
    return cl, pos, pseudo.nonlocal_tables(cl, pos, _psp()), V


def _bounds(cl, tab, V):
    """Spectral bounds: FD kinetic maximum + potential + the largest nonlocal eigenvalue of one atom."""
    st = _stencil(cl)
    kin = -0.5 * float(_lap_symbol(cl, st, np.zeros(3)).min())
    a0 = tab.img_atom == 0
    off = np.concatenate([[0], np.cumsum(tab.img_ndc.astype(np.int64) * tab.atom_nproj[tab.img_atom])])
    npj = int(tab.atom_nproj[0])
    chi = np.concatenate([tab.chi[off[i]:off[i + 1]].reshape(npj, -1) for i in np.nonzero(a0)[0]], axis=1)
    nl = np.linalg.eigvals(cl.dV * (chi @ chi.T) * tab.gamma[None, :npj]).real
    return float(V.min()) - 0.5, kin + float(V.max()) + 1.2 * max(0.0, float(nl.max())) + 0.5


def _orbitals(nd, ncol, seed, cplx):
    """Start orbitals of an SCF run: uniform(-1/2, 1/2)."""
    x = torch.rand(ncol, nd * (2 if cplx else 1), device=DEV, dtype=torch.float64, generator=_rng(seed)) - 0.5
    return torch.view_as_complex(x.view(ncol, nd, 2)) if cplx else x


def _smooth_orbitals(cl, ncol, seed, cplx):
    """Normalised orbitals with a plane-wave spectrum that falls off, as converged ones have."""
    nx, ny, nz = cl.shape
    k2 = 0.0
    for n, L, s in ((nz, cl.lengths[2], (-1, 1, 1)), (ny, cl.lengths[1], (1, -1, 1)), (nx, cl.lengths[0], (1, 1, -1))):
        k2 = k2 + (2 * math.pi / L * n * torch.fft.fftfreq(n, device=DEV, dtype=torch.float64)).view(s) ** 2
    c = torch.randn(ncol, nz, ny, nx, device=DEV, dtype=torch.complex128, generator=_rng(seed)) * torch.exp(-0.5 * k2)
    x = torch.fft.ifftn(c, dim=(1, 2, 3)).reshape(ncol, -1)
    x = x if cplx else x.real.contiguous()
    return x / (x.norm(dim=1, keepdim=True) * math.sqrt(cl.dV))


def _kpoint(cl):
    return np.array([0.25, 0.125, -0.375]) * 2 * math.pi / cl.lengths


def _context(cl, tab, kcart=None):
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    if kcart is not None:
        ctx.set_kpoint(kcart)
    return ctx


def _problems(case, seed):
    """The independent problems of a batch: (cell, tables, V, k-point or None, weight, orbitals)."""
    out = []
    g = case["grid"]
    cl, _, tab, V = _system({"reps": 0, "shape": f"{g}x{g}x{g}"}, seed)
    kc, _, w = C.kpoints_mp(cl, [case["kgrid"]] * 3)
    for i in range(len(kc)):
        out.append((cl, tab, V, kc[i], float(w[i]) / float(w.sum()), _orbitals(cl.nd, case["ncol"], seed + i, True)))
    r = np.random.default_rng(seed)
    for i, g in enumerate(_cells(case)):
        cl, _, tab, V = _system({"reps": 1, "shape": f"{g}x{g}x{g}"}, seed + 100 + i, strain=float(r.uniform(-0.03, 0.03)))
        out.append((cl, tab, V, None, 1.0, _orbitals(cl.nd, case["ncol_cell"], seed + 200 + i, False)))
    return out


def _inputs(case, seed):
    """The inputs of a case, made from the seed alone and without a context."""
    kind = case["kind"]
    if kind == "batch":
        return {"problems": _problems(case, seed)}
    cl, pos, tab, V = _system(case, seed)
    kpt = bool(case.get("kpt"))
    s = {"cell": cl, "tab": tab, "V": V, "kcart": _kpoint(cl) if kpt else None, "kpt": kpt}
    if kind in ("filter", "pass"):
        lo, hi = _bounds(cl, tab, V)
        s.update(lc=0.5 * (lo + hi), lo=lo, hi=hi)
    if kind == "veff":
        q = (2 * math.pi) ** 1.5
        s["rho"] = 0.004 + 4.0 / (q * 1.6 ** 3) * _gaussians(cl, pos, 1.6)
        s["rho_b"] = -4.0 / (q * 0.8 ** 3) * _gaussians(cl, pos, 0.8)
    elif kind == "forces":
        s["psi"] = _smooth_orbitals(cl, case["ncol"], seed, kpt)
        n = np.arange(case["ncol"])
        s["occ"] = 1.0 / (1.0 + np.exp((n - 0.8 * case["ncol"]) / 2.0))
    else:
        s["psi"] = _orbitals(cl.nd, case["ncol"], seed, kpt)
    if kind == "autograd":
        s["grad"] = _orbitals(cl.nd, case["ncol"], seed + 1, False)
    if kind == "pass":
        s["nelectron"] = 4.0 * len(pos)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "batch":
        s["solvers"] = [solver.EigenSolver(_context(cl, tab, k), case["precision"])
                        for cl, tab, _, k, _, _ in s["problems"]]
        s["psis"] = [p[5] for p in s["problems"]]
        b = [_bounds(p[0], p[1], p[2]) for p in s["problems"]]
        s["lo"], s["hi"] = [x[0] for x in b], [x[1] for x in b]
        s["lc"] = [0.5 * (x[0] + x[1]) for x in b]
        # the program has used every context before (here: one filter step of one orbital), so the
        # layouts that a context makes once of its projector tables are in place
        for i, (es, p) in enumerate(zip(s["solvers"], s["problems"])):
            es.chebyshev_filter(p[5][:1], p[2], s["lc"][i], s["lo"][i], s["hi"][i], degree=1, kpt=p[3] is not None)
        return s
    s["ctx"] = _context(s["cell"], s["tab"], s["kcart"])
    if case["kind"] in ("filter", "pass"):
        s["solver"] = solver.EigenSolver(s["ctx"], case["precision"])
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_apply(s):
    h = solver.Hamiltonian(s["ctx"])
    return h.apply_kpt(s["psi"], Veff=s["V"]) if s["kpt"] else h.apply(s["psi"], Veff=s["V"])


def _run_autograd(s):
    psi, V = s["psi"].detach().requires_grad_(True), s["V"].detach().requires_grad_(True)
    y = autograd.hamiltonian_apply(s["ctx"], psi, V)
    gp, gv = torch.autograd.grad(y, (psi, V), s["grad"])
    return {"y": y.detach(), "grad_psi": gp, "grad_veff": gv}


def _run_filter(s):
    return s["solver"].chebyshev_filter(s["psi"], s["V"], s["lc"], s["lo"], s["hi"], degree=s["case"]["degree"],
                                        kpt=s["kpt"])


def _run_pass(s):
    """One SCF iteration's eigensolver and density; bounds move on from pass to pass as in the SCF
    loop.  The orbitals themselves are defined up to signs and mixing of close states, so what
    comes back of them is what the loop uses: the Ritz values, the Fermi level and the density."""
    es = s["solver"]
    _, eig, rho, _ = es.solve_density(s["psi"], s["V"], s["lc"], s["lo"], s["hi"], 20, nelectron=s["nelectron"],
                                       beta=BETA)
    s["lc"], s["lo"] = es.lambda_cutoff(), float(eig[0])
    return {"eig": eig, "rho": rho}


def _run_batch(s):
    """One CheFSI pass over every problem, then the density of the k-point cell (one Fermi level over
    its k-points) and of every other cell."""
    prob, es = s["problems"], s["solvers"]
    kpt = [p[3] is not None for p in prob]
    res = solver.solve_batch(es, s["psis"], [p[2] for p in prob], s["lc"], s["lo"], s["hi"], 20, kpt=kpt)
    s["lc"], s["lo"] = [e.lambda_cutoff() for e in es], [float(r[1][0]) for r in res]
    ks = [i for i, k in enumerate(kpt) if k]
    n = len(res[ks[0]][1])
    ef = solver.fermi_level(np.concatenate([res[i][1] for i in ks]),
                            np.concatenate([np.full(n, 2.0 * prob[i][4]) for i in ks]), 8.0, BETA)
    rho = None
    for i in ks:
        rho = solver.electron_density(es[i].ctx, res[i][0], solver.occupations(res[i][1], ef, BETA), 2.0 * prob[i][4],
                                      rho, True)
    out = {"eig": [r[1] for r in res], "rho": [rho]}
    for i in range(len(ks), len(prob)):
        e = solver.fermi_level(res[i][1], np.full(len(res[i][1]), 2.0), 32.0, BETA)
        out["rho"].append(solver.electron_density(es[i].ctx, res[i][0], solver.occupations(res[i][1], e, BETA)))
    return out


def _run_veff(s):
    r = EffectivePotential(s["ctx"]).compute(s["rho"], s["rho_b"])
    return {"veff": r.veff, "vxc": r.vxc, "exc": r.exc, "phi": r.phi}


def _run_forces(s):
    nl = solver.NonlocalProjector(s["ctx"])
    f, e = nl.force(s["psi"], s["occ"], kpt=s["kpt"])
    sk, snl = nl.stress(s["psi"], s["occ"], kpt=s["kpt"])
    return {"force": f, "energy": e, "stress_k": sk, "stress_nl": snl}


_RUN = {"apply": _run_apply, "autograd": _run_autograd, "filter": _run_filter, "pass": _run_pass, "batch": _run_batch,
        "veff": _run_veff, "forces": _run_forces}


# ---------------------------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------------------------
def _work_solve(nd, n, cplx, degree, rr):
    """Orbitals in and out once, V once; the degree-m recurrence (6 * 6 neighbours, centre, V, x_old:
    about 80 operations a real number and step), Gram products and rotation."""
    c = 2 if cplx else 1
    f = 80.0 * nd * n * c * degree
    if rr:
        f += 2.0 * nd * n * n * (4 if cplx else 1) * 2.5 + 80.0 * nd * n * c
    return 16.0 * nd * n * c + 8.0 * nd, f


def work(case):
    kind = case["kind"]
    if kind == "batch":
        nk = {1: 1, 2: 8, 3: 14}[case["kgrid"]]
        parts = [_work_solve(case["grid"] ** 3, case["ncol"], True, 20, True)] * nk
        parts += [_work_solve(g ** 3, case["ncol_cell"], False, 20, True) for g in _cells(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    nd = float(np.prod(_shape(case)))
    if kind == "veff":
        return {"bytes": 8.0 * nd * 6, "flops": nd * (6 * 24 + 600 + 60 * math.log2(nd))}
    n, c = case["ncol"], 2 if case.get("kpt") else 1
    if kind == "apply":
        return {"bytes": 8.0 * nd * (2 * n * c + 1), "flops": 80.0 * nd * n * c}
    if kind == "autograd":
        return {"bytes": 8.0 * nd * (4 * n + 2), "flops": 162.0 * nd * n}
    if kind == "forces":
        return {"bytes": 8.0 * nd * n * c, "flops": nd * n * c * (3 * 24 + 12)}
    b, f = _work_solve(nd, n, c == 2, case["degree"] if kind == "filter" else 20, kind == "pass")
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the distance to exact() and between orders of summation, measured over the
    ranges (relative to it: apply 7e-16, 64-bit filter 1e-15, mixed filter 2e-7, 64-bit pass 2e-14,
    mixed pass 3e-7, potential 2e-14, forces 2e-15), wider where a Ritz value's error acts on the
    occupation of a state at the Fermi level (times the inverse smearing)."""
    kind = case["kind"]
    if kind in ("apply", "autograd"):
        return {"rel": 1e-14, "max": 1e-12}
    if kind in ("veff", "forces"):
        return {"rel": 1e-12, "max": 1e-10}
    if kind == "filter":
        return {"rel": 1e-6, "max": 4e-5} if case["precision"] == "mixed" else {"rel": 1e-13, "max": 1e-11}
    return {"rel": 2e-5, "max": 1e-3} if case["precision"] == "mixed" else {"rel": 1e-10, "max": 1e-8}


# ---------------------------------------------------------------------------------------------
# 64-bit values in plain torch.  Periodic FD operators are convolutions: multiplication by their
# symbol in Fourier space (Bloch functions: at angles shifted by the phase of one cell).
# ---------------------------------------------------------------------------------------------
def _stencil(cl):
    r = cl.fd_order // 2
    w1, w2 = np.zeros(r + 1), np.zeros(r + 1)
    for p in range(1, r + 1):
        f = 1.0
        for q in range(r - p + 1, r + 1):
            f *= q
        for q in range(r + 1, r + p + 1):
            f /= q
        w1[p] = (-1) ** (p + 1) * f / p
        w2[p] = 2 * (-1) ** (p + 1) * f / (p * p)
        w2[0] -= 2.0 / (p * p)
    return w1, w2


def _angles(cl, kcart, d):
    n = cl.shape[d]
    return (2 * math.pi * n * torch.fft.fftfreq(n, device=DEV, dtype=torch.float64)
            + float(kcart[d] * cl.lengths[d])) / n


def _on_axis(t, d):
    return t.view([(-1, 1, 1), (1, -1, 1), (1, 1, -1)][2 - d])


def _d1_symbol(cl, st, kcart, d):
    """First derivative along lattice direction d: i times this."""
    a, h = _angles(cl, kcart, d), float(cl.spacing[d])
    return _on_axis(sum(2.0 * float(st[0][p]) / h * torch.sin(p * a) for p in range(1, len(st[0]))), d)


def _lap_symbol(cl, st, kcart):
    T = np.eye(3) if cl.orthogonal else cl.lapc_T
    out = 0.0
    for d in range(3):
        a, h = _angles(cl, kcart, d), float(cl.spacing[d])
        s = float(st[1][0]) + sum(2.0 * float(st[1][p]) * torch.cos(p * a) for p in range(1, len(st[1])))
        out = out + _on_axis(float(T[d, d]) / (h * h) * s, d)
    if not cl.orthogonal:
        g = [_d1_symbol(cl, st, kcart, d) for d in range(3)]
        for a, b in ((0, 1), (0, 2), (1, 2)):
            out = out - 2.0 * float(T[a, b]) * g[a] * g[b]
    return out


class _Exact:
    """H psi, projections and FD derivatives in 64 bits for one cell and k-point."""

    def __init__(self, cl, tab, V, kcart=None):
        self.cl, self.V = cl, V
        self.cplx = kcart is not None
        self.k = np.zeros(3) if kcart is None else np.asarray(kcart)
        self.st = _stencil(cl)
        self.lap = _lap_symbol(cl, self.st, self.k)
        nx, ny, nz = cl.shape
        self.grid = (nz, ny, nx)
        if self.cplx:
            ph = 0.0
            for d, n in enumerate(cl.shape):
                t = torch.arange(n, device=DEV, dtype=torch.float64) * (float(self.k[d] * cl.lengths[d]) / n)
                ph = ph + _on_axis(t, d)
            self.bloch = torch.polar(torch.ones_like(ph), ph)
        self._tables(tab)

    def _tables(self, tab):
        """Per atom: all points of its images, the projector values there (Bloch factor included),
        padded to the largest atom with zeros."""
        na, npj = tab.n_atom, int(tab.atom_nproj[0])
        go = np.concatenate([[0], np.cumsum(tab.img_ndc)])
        per = [np.nonzero(tab.img_atom == a)[0] for a in range(na)]
        m = max(int(tab.img_ndc[p].sum()) for p in per)
        idx, chi = np.zeros((na, m), np.int64), np.zeros((na, m, npj), np.complex128)
        rel = np.zeros((na, m, 3))
        nx, ny, _ = self.cl.shape
        for a in range(na):
            o = 0
            for i in per[a]:
                n, g = int(tab.img_ndc[i]), tab.gpos[go[i]:go[i + 1]].astype(np.int64)
                idx[a, o:o + n] = g
                ph = np.exp(-1j * float(self.k @ tab.img_shift[i]))
                chi[a, o:o + n] = ph * tab.chi[go[i] * npj:go[i + 1] * npj].reshape(npj, n).T
                ijk = np.stack([g % nx, g // nx % ny, g // (nx * ny)], 1) * self.cl.spacing - tab.img_coords[i]
                rel[a, o:o + n] = ijk if self.cl.orthogonal else ijk @ self.cl.uvec
                o += n
        self.idx = torch.from_numpy(idx).to(DEV)
        self.rel = torch.from_numpy(rel).to(DEV)
        self.chi = torch.from_numpy(chi if self.cplx else chi.real.copy()).to(DEV)
        self.gam = torch.from_numpy(tab.gamma.reshape(na, npj)).to(DEV).to(self.chi.dtype)

    def _convolve(self, x, symbol):
        y = x.view(-1, *self.grid)
        if self.cplx:
            y = torch.fft.ifftn(torch.fft.fftn(y * self.bloch.conj(), dim=(1, 2, 3)) * symbol, dim=(1, 2, 3)) * self.bloch
        else:
            h = self.grid[2] // 2 + 1
            y = torch.fft.irfftn(torch.fft.rfftn(y, dim=(1, 2, 3)) * symbol[..., :h], s=self.grid, dim=(1, 2, 3))
        return y.reshape(x.shape)

    def project(self, x, weight=None):
        """dV chi^T x per column, atom and projector."""
        c = self.chi if weight is None else self.chi * weight[..., None]
        return self.cl.dV * torch.einsum("nam,amp->nap", x[:, self.idx], c)

    def h(self, x):
        y = torch.cat([-0.5 * self._convolve(b, self.lap) for b in x.split(64)])
        y += self.V * x
        add = torch.einsum("nap,amp->nam", self.gam * self.project(x), self.chi.conj())
        return y.index_add_(1, self.idx.reshape(-1), add.reshape(len(x), -1))

    def grad(self, x, d):
        """FD derivative along lattice direction d."""
        s = _d1_symbol(self.cl, self.st, self.k, d) * 1j
        if not self.cplx and self.cl.shape[d] % 2 == 0:  # the highest mode has no odd part
            s.select(2 - d, self.cl.shape[d] // 2).zero_()
        return self._convolve(x, s)

    def filter(self, x, lc, lo, hi, degree):
        e, c = (hi - lc) / 2, (hi + lc) / 2
        s1 = s = e / (lo - c)
        y = (s1 / e) * (self.h(x) - c * x)
        for _ in range(2, degree + 1):
            sn = 1.0 / (2.0 / s1 - s)
            x, y = y, (2 * sn / e) * (self.h(y) - c * y) - s * sn * x
            s = sn
        return y

    def solve(self, x, lc, lo, hi, degree):
        y = self.filter(x, lc, lo, hi, degree)
        y = y / y.abs().max()
        hy = self.h(y)
        m, hs = y.conj() @ y.T * self.cl.dV, y.conj() @ hy.T * self.cl.dV
        inv = torch.linalg.inv(torch.linalg.cholesky(0.5 * (m + m.mH)))
        e, q = torch.linalg.eigh(inv @ (0.5 * (hs + hs.mH)) @ inv.mH)
        return e, (inv.mH @ q).T @ y


def _fermi(eig, w, ne):
    lo, hi = eig.min() - 1.0, eig.max() + 1.0
    for _ in range(200):
        m = 0.5 * (lo + hi)
        if (w * _occ(eig, m)).sum() > ne:
            hi = m
        else:
            lo = m
    return 0.5 * (lo + hi)


def _occ(eig, ef):
    return 1.0 / (1.0 + np.exp(np.clip((eig - ef) * BETA, -700, 700)))


def _density(psi, w):
    w = torch.from_numpy(w).to(DEV)
    return sum((w[i:i + 64, None] * psi[i:i + 64].abs() ** 2).sum(0) for i in range(0, len(w), 64))


def _pbe(rho, sigma):
    """rho eps_xc of spin-unpolarised PBE (Perdew, Burke, Ernzerhof 1996; Perdew, Wang 1992)."""
    kappa, beta, gam = 0.804, 0.06672455060314922, (1 - math.log(2)) / math.pi ** 2
    r13 = rho ** (1.0 / 3.0)
    kf = (3 * math.pi ** 2) ** (1.0 / 3.0) * r13
    s2 = sigma / (2 * kf * rho) ** 2
    ex = -0.75 * (3 / math.pi) ** (1.0 / 3.0) * r13
    fx = 1 + kappa - kappa / (1 + beta * math.pi ** 2 / 3 * s2 / kappa)
    rs = (3 / (4 * math.pi)) ** (1.0 / 3.0) / r13
    g = 2 * 0.0310907 * (7.5957 * rs ** 0.5 + 3.5876 * rs + 1.6382 * rs ** 1.5 + 0.49294 * rs * rs)
    ec = -2 * 0.0310907 * (1 + 0.21370 * rs) * torch.log1p(1 / g)
    t2 = sigma * math.pi / (16 * kf * rho * rho)
    a = beta / gam / torch.expm1(-ec / gam) * t2
    return rho * (ex * fx + ec + gam * torch.log1p(beta / gam * t2 * (1 + a) / (1 + a + a * a)))


def _exact_veff(s):
    ex = _Exact(s["cell"], s["tab"], s["V"])
    rho = s["rho"].clone().requires_grad_(True)
    g = [ex.grad(s["rho"][None], d)[0] for d in range(3)]
    sigma = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2).requires_grad_(True)
    f = _pbe(rho, sigma)
    vr, vs = torch.autograd.grad(f.sum(), (rho, sigma))
    vxc = vr - sum(ex.grad((2 * vs * g[d])[None], d)[0] for d in range(3))
    b = 4 * math.pi * (s["rho"] + s["rho_b"])
    b = b - b.mean()
    sym = -ex.lap[..., :ex.grid[2] // 2 + 1]
    sym = torch.where(sym.abs() < 1e-12, torch.inf, sym)
    phi = torch.fft.irfftn(torch.fft.rfftn(b.view(ex.grid)) / sym, s=ex.grid).reshape(-1)
    phi = phi - phi.mean()
    return {"veff": vxc + phi, "vxc": vxc, "exc": (f / rho).detach(), "phi": phi}


def _exact_forces(s):
    cl = s["cell"]
    ex = _Exact(cl, s["tab"], s["V"], s["kcart"])
    occ = torch.from_numpy(s["occ"]).to(DEV)
    of = 2.0
    gam = ex.gam.real
    al = ex.project(s["psi"])
    g = [ex.grad(s["psi"], d) for d in range(3)]

    def pair(u, v):
        return torch.einsum("n,ap,nap->a", occ, gam, (u.conj() * v).real)

    force = torch.stack([-2 * of * pair(al, ex.project(g[d])) for d in range(3)], 1)
    energy = float(of * pair(al, al).sum())
    if not cl.orthogonal:
        ui = torch.from_numpy(np.linalg.inv(cl.uvec)).to(DEV)
        g = [sum(ui[d, e] * g[e] for e in range(3)) for d in range(3)]
    sk, snl = [], []
    for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)):
        sk.append(-of * cl.dV * float((occ * (g[a].conj() * g[b]).real.sum(1)).sum()))
        snl.append(-2 * of * float(pair(al, ex.project(g[a], ex.rel[..., b])).sum()) - (energy if a == b else 0.0))
    return {"force": force.cpu().numpy(), "energy": energy, "stress_k": np.array(sk), "stress_nl": np.array(snl)}


def exact(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    if kind == "veff":
        return _exact_veff(s)
    if kind == "forces":
        return _exact_forces(s)
    if kind == "batch":
        eig, psis = [], []
        for cl, tab, V, k, _, psi in s["problems"]:
            lo, hi = _bounds(cl, tab, V)
            e, p = _Exact(cl, tab, V, k).solve(psi, 0.5 * (lo + hi), lo, hi, 20)
            eig.append(e.cpu().numpy())
            psis.append(p)
        ks = [i for i, p in enumerate(s["problems"]) if p[3] is not None]
        w = [2.0 * s["problems"][i][4] for i in ks]
        ef = _fermi(np.concatenate([eig[i] for i in ks]), np.repeat(w, len(eig[0])), 8.0)
        rho = [sum(_density(psis[i], w[i] * _occ(eig[i], ef)) for i in ks)]
        for i in range(len(ks), len(eig)):
            e = _fermi(eig[i], np.full(len(eig[i]), 2.0), 32.0)
            rho.append(_density(psis[i], 2.0 * _occ(eig[i], e)))
        return {"eig": eig, "rho": rho}
    ex = _Exact(s["cell"], s["tab"], s["V"], s["kcart"])
    if kind == "apply":
        return ex.h(s["psi"])
    if kind == "autograd":
        return {"y": ex.h(s["psi"]), "grad_psi": ex.h(s["grad"]), "grad_veff": (s["grad"] * s["psi"]).sum(0)}
    if kind == "filter":
        return ex.filter(s["psi"], s["lc"], s["lo"], s["hi"], case["degree"])
    e, psi = ex.solve(s["psi"], s["lc"], s["lo"], s["hi"], 20)
    e = e.cpu().numpy()
    ef = _fermi(e, np.full(len(e), 2.0), s["nelectron"])
    return {"eig": e, "rho": _density(psi, 2.0 * _occ(e, ef))}
