"""Odd nx in the pipelined stencil (padded rows, element-wise wrapped x neighbours) against the numpy
oracle, rows that end one or two points past a thread block, with and without the fused nonlocal term;
and the mixed pass, whose products stay FP64 for odd nx."""
import numpy as np
import pytest

from lynx_b200 import _lib
from lynx_b200 import cell as C
from lynx_b200 import pseudo as P
from oracle import chefsi_oracle as O

pytestmark = pytest.mark.gpu


def _system(synth_psp8, reps, shape):
    from lynx_b200 import solver
    cl, pos = C.diamond_si(reps, shape, displace=0.02, seed=9)
    V = C.synthetic_veff_separable(cl, pos, noise=1e-3, seed=9)
    tab = P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8))
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    t = dict(img_atom=tab.img_atom, img_ndc=tab.img_ndc, img_shift=tab.img_shift, gpos=tab.gpos, chi=tab.chi,
             gamma=tab.gamma, nproj=int(tab.atom_nproj[0]))
    return solver, ctx, V, O.Operator(cl.latvec, cl.shape, 12, True, t)


# FP64: 3 steps of sums of 60 terms; FP32: the same at 2^-24 per operation (measured 1e-6 of the largest)
@pytest.mark.parametrize("shape", [(49, 50, 52), (51, 48, 49), (53, 51, 50), (55, 49, 48)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-5)])
@pytest.mark.parametrize("fuse", [1, 0])
def test_filter(synth_psp8, shape, precision, tol, fuse):
    solver, ctx, V, H = _system(synth_psp8, 2, shape)
    ctx.set_option(_lib.OPT_FUSE_NONLOCAL, fuse)
    x = C.random_orbitals(ctx.nd, 3, seed=2)
    y = solver.EigenSolver(ctx, precision).chebyshev_filter(x, V, 25.0, -2.0, 70.0, degree=3)
    want = O.chebyshev_filter(H, x, V, 25.0, -2.0, 70.0, 3)
    assert np.abs(y - want).max() < tol * np.abs(want).max()
    ctx.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape", [(117, 48, 16), (237, 40, 12), (239, 20, 16)])
def test_densely_packed_spheres(shape, precision):
    """Every grid point in a sphere: a band's expanded values take as much shared memory as its rows, and
    the bands are made shorter until the stages fit.  Bitwise the separate nonlocal term."""
    from lynx_b200 import solver
    cl = C.Cell(np.diag([n * 0.35 for n in shape]), shape)
    nat, r = 36, np.random.default_rng(7)
    gpos = np.arange(cl.nd, dtype=np.int32)
    ndc = np.diff(np.linspace(0, cl.nd, nat + 1).astype(np.int32)).astype(np.int32)
    tab = P.NonlocalTables(np.arange(nat, dtype=np.int32), ndc, np.zeros((nat, 3)), np.zeros((nat, 3)), gpos,
                           r.normal(size=2 * cl.nd), np.full(nat, 2, np.int32), 1e-3 * r.normal(size=2 * nat))
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    V = r.normal(size=cl.nd)
    x = C.random_orbitals(ctx.nd, 40, seed=3)
    out = []
    for fuse in (1, 0):
        ctx.set_option(_lib.OPT_FUSE_NONLOCAL, fuse)
        out.append(solver.EigenSolver(ctx, precision).chebyshev_filter(x, V, 25.0, -9.0, 75.0, degree=3))
    assert np.array_equal(out[0], out[1])
    ctx.close()


@pytest.mark.parametrize("n", [41, 130])
def test_mixed_pass(synth_psp8, n):
    """The products of odd rows are FP64 products of the filtered block with and without the tensor-core
    option, bitwise; orthonormal orbitals, and the density that comes with the pass is theirs."""
    import torch
    solver, ctx, V, _ = _system(synth_psp8, 1, (25, 26, 27))
    es = solver.EigenSolver(ctx, "mixed")
    x = np.ascontiguousarray(C.random_orbitals(ctx.nd, n, seed=3).T)
    lo, hi = float(V.min()) - 1.0, ctx.max_eigval_half_lap + 8.0
    out = []
    for tc in (1, 0):
        ctx.set_option(_lib.OPT_TC_RAYLEIGH_RITZ, tc)
        psi = torch.from_numpy(x).cuda()
        _, eig, rho, ef = es.solve_density(psi, V, 0.5 * (lo + hi), lo, hi, 8, nelectron=32.0)
        w = solver.electron_density(ctx, psi, solver.occupations(eig, ef, 1000.0))
        assert float((rho - w).abs().max()) < 1e-12 * float(w.abs().max())
        s = (psi @ psi.T).cpu().numpy() * ctx.dV
        assert np.abs(s - np.eye(n)).max() < 1e-12
        out.append((eig, psi.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    ctx.close()


def test_mixed_kpt_pass(synth_psp8):
    solver, ctx, V, _ = _system(synth_psp8, 1, (25, 24, 23))
    ctx.set_kpoint(np.array([0.25, -0.125, 0.375]) * 2 * np.pi / ctx.cell.lengths)
    es = solver.EigenSolver(ctx, "mixed")
    lo, hi = float(V.min()) - 1.0, ctx.max_eigval_half_lap + 8.0
    out = []
    for tc in (1, 0):
        ctx.set_option(_lib.OPT_TC_RAYLEIGH_RITZ, tc)
        x = C.random_orbitals(ctx.nd, 45, seed=3, complex_=True)
        out.append(es.solve_kpt(x, V, 0.5 * (lo + hi), lo, hi, 6))
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][0], out[1][0])
    ctx.close()
