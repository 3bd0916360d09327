"""Kernels of small problems: the one-thread-per-point stencil, the one-kernel nonlocal apply of few
atoms, and the four-launch Rayleigh-Ritz step of few states, against the numpy oracle, the pipelined
stencil and dense linear algebra."""
import dataclasses

import numpy as np
import pytest

from helpers import si8_small
from lynx_b200 import _lib
from lynx_b200 import cell as C
from lynx_b200 import pseudo as P
from oracle import chefsi_oracle as O

pytestmark = pytest.mark.gpu


def _oracle(cl, tab):
    t = dict(img_atom=tab.img_atom, img_ndc=tab.img_ndc, img_shift=tab.img_shift, gpos=tab.gpos, chi=tab.chi,
             gamma=tab.gamma, nproj=int(tab.atom_nproj[0]))
    return O.Operator(cl.latvec, cl.shape, cl.fd_order, cl.orthogonal, t)


def _cell(kind, shape):
    if kind == "fcc":
        cl, pos = C.fcc_si_primitive(shape[0])
        cl.shape = shape
        return cl, pos, C.synthetic_veff(cl, pos, noise=1e-3, seed=2)
    cl, pos, V = si8_small(grid=shape)
    return cl, pos, V


# FP64: sums of about 60 terms of size ~40 |x| (coefficients / h^2): 60 * 2^-53 * 40 / |H x| < 1e-13.
@pytest.mark.parametrize("kind,shape,ncol,kpt", [
    ("si8", (20, 21, 22), 1, False), ("si8", (21, 20, 23), 3, False), ("si8", (20, 20, 20), 25, False),
    ("si8", (20, 21, 22), 5, True), ("si8", (31, 33, 30), 2, True), ("fcc", (20, 20, 20), 4, False),
    ("fcc", (17, 19, 18), 3, True)])
@pytest.mark.parametrize("fd_order", [12, 8])
def test_h_apply_of_small_blocks(synth_psp8, kind, shape, ncol, kpt, fd_order):
    from lynx_b200 import solver
    cl, pos, V = _cell(kind, shape)
    cl.fd_order = fd_order
    tab = P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8))
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    k = np.array([0.25, -0.125, 0.375]) * 2 * np.pi / cl.lengths
    x = C.random_orbitals(ctx.nd, ncol, seed=3, complex_=kpt)
    h = solver.Hamiltonian(ctx, V)
    if kpt:
        ctx.set_kpoint(k)
        y = h.apply_kpt(x)
    else:
        y = h.apply(x)
    want = _oracle(cl, tab).apply(x, V, kpt=k if kpt else None)
    assert np.abs(y - want).max() < 1e-12 * np.abs(want).max()
    ctx.close()


def test_complex_projections_of_very_many_atoms():
    """70000 one-point atoms, above the extent of a grid in y, every other of the later ones without a
    projector: the nonlocal term is then a factor per grid point (1e-14: sums of about 8 terms)."""
    from lynx_b200 import solver
    cl, _, _ = _cell("si8", (20, 21, 22))
    n, r = 70000, np.random.default_rng(5)
    nproj = np.ones(n, np.int32)
    nproj[65535::2] = 0
    chi, gamma, gpos = r.normal(size=nproj.sum()), r.normal(size=nproj.sum()), r.integers(0, cl.nd, n)
    tab = P.NonlocalTables(np.arange(n, dtype=np.int32), np.ones(n, np.int32), np.zeros((n, 3)), np.zeros((n, 3)),
                           gpos.astype(np.int32), chi, nproj, gamma)
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    x = C.random_orbitals(ctx.nd, 2, seed=4, complex_=True)
    got = solver.NonlocalProjector(ctx).apply(x, np.zeros_like(x), kpt=True)
    f = np.bincount(gpos[nproj > 0], weights=chi * chi * gamma * cl.dV, minlength=cl.nd)
    assert np.abs(got - f[:, None] * x).max() < 1e-14 * np.abs(f).max()
    ctx.close()


def _launches(ctx, f):
    ctx.lib.lynx_launch_count(1)
    out = f()
    return out, ctx.lib.lynx_launch_count(0)


@pytest.mark.parametrize("ncol", [3, 40])  # below and above 1.25 MB in both precisions
@pytest.mark.parametrize("kind", ["dirichlet", "dirichlet-odd", "fcc"])
def test_both_stencils_of_phased_and_skewed_cells(synth_psp8, kind, ncol):
    """Dirichlet directions (zero ghosts) and real blocks of a non-orthogonal cell, with the direct step and
    with the pipelined kernel (and the separate derivative kernels of the skewed cell): H psi and both
    filters against the oracle.  Tolerances as for the periodic cells: 1e-12, 1e-10, 2e-5."""
    from lynx_b200 import solver
    if kind == "fcc":
        cl, pos, V = _cell("fcc", (20, 20, 20))
        tab = P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8))
        H = _oracle(cl, tab)
    else:
        shape = (20, 22, 24) if kind == "dirichlet" else (21, 22, 20)
        cl = C.Cell(C.diamond_si(1, 20)[0].latvec, shape, True, (1, 0, 1), 12)
        V, tab = np.random.default_rng(4).normal(size=cl.nd), None
        H = O.Operator(cl.latvec, cl.shape, order=12, orthogonal=True, bc=cl.bc)
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    x = C.random_orbitals(ctx.nd, ncol, seed=91)
    y, want = solver.Hamiltonian(ctx, V).apply(x, shift=0.3), H.apply(x, V, 0.3)
    assert np.abs(y - want).max() < 1e-12 * np.abs(want).max()
    bounds = (25.0, -2.0, ctx.max_eigval_half_lap + 4.0)
    want = O.chebyshev_filter(H, x, V, *bounds, 3)
    es = solver.EigenSolver(ctx)
    for prec, tol in (("fp64", 1e-10), ("mixed", 2e-5)):
        y = es.chebyshev_filter(x, V, *bounds, 3, precision=prec)
        assert np.abs(y - want).max() < tol * np.abs(want).max()
    ctx.close()


@pytest.mark.parametrize("nx", [512, 514, 608])
def test_small_blocks_of_long_rows(nx):
    """Rows that the direct step does not take (above 512) run the pipelined kernel, small block or not."""
    from lynx_b200 import solver
    cl = C.Cell(np.diag([nx * 0.35, 5.0, 5.5]), (nx, 14, 16))
    V = np.random.default_rng(2).normal(size=cl.nd)
    x = C.random_orbitals(cl.nd, 1, seed=3)
    ctx = solver.Context(cl)
    y = solver.Hamiltonian(ctx, V).apply(x)
    want = O.Operator(cl.latvec, cl.shape).apply(x, V)
    assert np.abs(y - want).max() < 1e-12 * np.abs(want).max()
    ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_atom_kernel_up_to_2048_pairs(synth_psp8, precision):
    """8 atoms: 256 columns take the one-kernel apply (two launches a degree), 257 the staged gather, the
    expansion and the fused term (three).  The same sums in another order: the columns agree to 100
    roundings of the largest value (2^-53, 2^-24), a degree-3 filter's growth included."""
    from lynx_b200 import solver
    cl, pos, V = _cell("si8", (20, 18, 20))
    ctx = solver.Context(cl)
    ctx.set_option(_lib.OPT_AUTOTUNE, 0)
    ctx.set_nonlocal(P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8)))
    es = solver.EigenSolver(ctx, precision)
    x = C.random_orbitals(ctx.nd, 257, seed=6)
    out = []
    for n, per_degree in ((256, 2), (257, 3)):
        f = lambda degree: es.chebyshev_filter(x[:, :n], V, 25.0, -2.0, 70.0, degree=degree)
        n1 = _launches(ctx, lambda: f(2))[1]
        y, n2 = _launches(ctx, lambda: f(3))
        assert n2 - n1 == per_degree
        out.append(y[:, :256])
    eps = 2.0 ** -53 if precision == "fp64" else 2.0 ** -24
    assert np.abs(out[0] - out[1]).max() < 100 * eps * np.abs(out[1]).max()
    ctx.close()


@pytest.mark.parametrize("block", [128, 37])
def test_column_blocks_of_a_host_solve_take_one_route(synth_psp8, block):
    """8 atoms and 300 columns are above the line, each block of the host solve's pipelined copy below it:
    the line is the whole block's, so the two solves agree bitwise."""
    import ctypes
    from lynx_b200 import solver
    cl, pos, V = _cell("si8", (20, 18, 20))
    ctx = solver.Context(cl)
    ctx.set_nonlocal(P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8)))
    n, lo, hi = 300, float(V.min()) - 1.0, ctx.max_eigval_half_lap + 8.0
    x = C.random_orbitals(ctx.nd, n, seed=7)
    want, e_want = solver.EigenSolver(ctx, "mixed").solve(x, V, 0.5 * (lo + hi), lo, hi, 5)
    got, eig, lc = np.asfortranarray(x.copy()), np.zeros(n), ctypes.c_double()
    ctx.set_option(_lib.OPT_HOST_COPY_BLOCK, block)
    _lib.check(ctx.lib.lynx_eigensolver_solve_host(ctx.handle, _lib.dptr(got), _lib.dptr(eig),
                                                   _lib.dptr(np.ascontiguousarray(V)), n, ctx.nd, 0.5 * (lo + hi), lo,
                                                   hi, 5, _lib.PREC_MIXED, ctypes.byref(lc)))
    assert np.array_equal(eig, e_want) and np.array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,ncol", [((20, 21, 22), 7), ((24, 24, 24), 1), ((22, 24, 26), 11)])
def test_direct_step_is_the_pipelined_one(synth_psp8, precision, shape, ncol):
    """The same sums in the same order: bitwise the pipelined kernel's filter (forced by the launch
    shape option).  All blocks below 1.25 MB in FP64, where the direct step is the default."""
    from lynx_b200 import solver
    cl, pos, V = _cell("si8", shape)
    ctx = solver.Context(cl)
    ctx.set_nonlocal(P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8)))
    es = solver.EigenSolver(ctx, precision)
    x = C.random_orbitals(ctx.nd, ncol, seed=4)
    out = []
    for forced in (0, 1):
        ctx.set_option(_lib.OPT_STENCIL_SHAPE, forced)
        out.append(es.chebyshev_filter(x, V, 25.0, -2.0, 70.0, degree=5))
    assert np.array_equal(out[0], out[1])
    ctx.close()


def _drop_projectors(tab, atoms):
    """The tables with the projectors of some atoms taken out; the atoms and their images stay."""
    lens = tab.img_ndc * tab.atom_nproj[tab.img_atom]
    keep = ~np.isin(tab.img_atom, atoms)
    chi = np.concatenate([b for b, k in zip(np.split(tab.chi, np.cumsum(lens)[:-1]), keep) if k] or [np.zeros(0)])
    nproj = tab.atom_nproj.copy()
    nproj[atoms] = 0
    gamma = np.concatenate([g for a, g in enumerate(np.split(tab.gamma, np.cumsum(tab.atom_nproj)[:-1]))
                            if a not in atoms] or [np.zeros(0)])
    return dataclasses.replace(tab, atom_nproj=nproj, chi=chi, gamma=gamma)


@pytest.mark.parametrize("kpt", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_atoms_without_projectors(synth_psp8, precision, kpt):
    """A filter with tables in which no atom has projectors is the filter without tables, bitwise; with
    every other atom left, H psi is the oracle's (1e-12 as above)."""
    from lynx_b200 import solver
    cl, pos, V = _cell("si8", (20, 21, 22))
    tab = P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8))
    ctx = solver.Context(cl)
    k = np.array([0.25, -0.125, 0.375]) * 2 * np.pi / cl.lengths
    ctx.set_kpoint(k)
    es = solver.EigenSolver(ctx, precision)
    x = C.random_orbitals(ctx.nd, 5, seed=4, complex_=kpt)
    out = []
    for t in (None, _drop_projectors(tab, np.arange(tab.n_atom))):
        ctx.set_nonlocal(t)
        out.append(es.chebyshev_filter(x, V, 25.0, -2.0, 70.0, degree=9, kpt=kpt))
    assert np.array_equal(out[0], out[1])
    drop = np.arange(0, tab.n_atom, 2)
    ctx.set_nonlocal(_drop_projectors(tab, drop))
    h = solver.Hamiltonian(ctx, V)
    gamma = tab.gamma.reshape(tab.n_atom, -1).copy()
    gamma[drop] = 0.0  # the oracle takes one projector count: no strength instead of no projector
    zero = dataclasses.replace(tab, gamma=gamma.ravel())
    want = _oracle(cl, zero).apply(x, V, kpt=k if kpt else None)
    got = h.apply_kpt(x) if kpt else h.apply(x)
    assert np.abs(got - want).max() < 1e-12 * np.abs(want).max()
    ctx.close()


@pytest.mark.parametrize("n", [1, 2, 3, 24, 39, 40, 41])
@pytest.mark.parametrize("kpt", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rayleigh_ritz_of_few_states(synth_psp8, n, kpt, precision):
    """One pass against dense linear algebra on the filtered block (n = 41: the library path).  FP64:
    eps times the condition of the overlap (a degree-4 filter: below 1e4).  Mixed: the FP32 filter."""
    from lynx_b200 import solver
    cl, pos, V = _cell("si8", (18, 17, 20))
    tab = P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8))
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    k = np.array([0.25, -0.125, 0.375]) * 2 * np.pi / cl.lengths if kpt else None
    if kpt:
        ctx.set_kpoint(k)
    lo, hi = float(V.min()) - 1.0, ctx.max_eigval_half_lap + 8.0
    x = C.random_orbitals(ctx.nd, n, seed=5, complex_=kpt)
    es = solver.EigenSolver(ctx, precision)
    psi, eig = (es.solve_kpt if kpt else es.solve)(x, V, 0.5 * (lo + hi), lo, hi, 4)
    want, e_want, _ = O.solve(_oracle(cl, tab), x, V, 0.5 * (lo + hi), lo, hi, 4, kpt=k)
    tol = 1e-11 if precision == "fp64" else 2e-5
    assert np.all(np.diff(eig) >= 0)
    assert np.abs(eig - e_want).max() < tol * np.abs(e_want).max()
    s = psi.conj().T @ psi * cl.dV
    assert np.abs(s - np.eye(n)).max() < (1e-11 if precision == "fp64" else 1e-5)
    sv = np.linalg.svd(psi.conj().T @ want * cl.dV, compute_uv=False)
    assert np.abs(sv - 1).max() < (1e-11 if precision == "fp64" else 1e-5)
    ctx.close()


@pytest.mark.parametrize("n", [4, 7])
def test_degenerate_states(n):
    """V = 0, no projectors, plane waves: the Ritz values of the cubic cell are degenerate in exact
    groups; the rotations must still converge and leave an orthonormal block."""
    from lynx_b200 import solver
    cl = C.diamond_si(1, 18)[0]
    ctx = solver.Context(cl)
    g = np.arange(18) * 2 * np.pi / 18
    zz, yy, xx = np.meshgrid(g, g, g, indexing="ij")
    waves = [np.ones(18 ** 3)] + [f(t).ravel() for t in (xx, yy, zz) for f in (np.cos, np.sin)]
    x = np.asfortranarray(np.stack(waves[:n], axis=1))
    hi = ctx.max_eigval_half_lap + 1.0
    psi, eig = solver.EigenSolver(ctx, "fp64").solve(x, np.zeros(ctx.nd), 0.5 * hi, -0.5, hi, 2)
    e1 = O.Operator(cl.latvec, cl.shape).apply(x[:, 1:2], np.zeros(ctx.nd))[5, 0] / x[5, 1]
    assert np.abs(eig - np.array([0.0] + [e1] * (n - 1))).max() < 1e-11
    assert np.abs(psi.T @ psi * cl.dV - np.eye(n)).max() < 1e-11
    ctx.close()


@pytest.mark.parametrize("kpt", [False, True])
@pytest.mark.parametrize("n", [5, 24])
def test_ritz_values_far_from_one(n, kpt):
    """H of size 2^-590 or 2^560, whose entries' squares leave the range of FP64.  A cell 2^300 times as
    wide is exactly 2^-600 of the same H; a potential of 2^560 against one of 2^100 leaves the kinetic term
    below rounding, so the values differ by 2^460 to the rounding of the products (about 1e3 terms)."""
    from lynx_b200 import solver
    cl = C.diamond_si(1, (15, 14, 16))[0]
    x = C.random_orbitals(cl.nd, n, seed=8, complex_=kpt)
    v = np.random.default_rng(3).normal(size=cl.nd)

    def ritz(scale, V, s):
        ctx = solver.Context(C.Cell(cl.latvec * scale, cl.shape))
        es = solver.EigenSolver(ctx, "fp64")
        _, eig = (es.solve_kpt if kpt else es.solve)(x, V, 25.0 * s, -9.0 * s, 70.0 * s, 1)
        ctx.close()
        return eig

    assert np.array_equal(ritz(2.0 ** 300, v * 2.0 ** -600, 2.0 ** -600), ritz(1.0, v, 1.0) * 2.0 ** -600)
    a, b = (ritz(1.0, v * 2.0 ** e, 2.0 ** e) for e in (100, 560))
    assert np.abs(b * 2.0 ** -460 - a).max() < 1e-12 * np.abs(a).max()
