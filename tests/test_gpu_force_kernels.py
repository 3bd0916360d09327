"""Nonlocal force and stress kernels on shapes other than the cubic ones: ragged grids, bands that do
not divide ny, several z chunks, rows longer than a block (the point-wise kinetic kernel), FD orders 12
and 8, one column; against the numpy oracle (sums of 1e6 terms in another order: 1e-11)."""
import numpy as np
import pytest

from lynx_b200 import cell as C
from lynx_b200 import pseudo as P
from oracle import chefsi_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape,ncol,kpt,order", [
    ("orth", (20, 21, 22), 1, False, 12), ("orth", (21, 35, 19), 3, True, 12), ("orth", (64, 13, 40), 2, False, 12),
    ("orth", (22, 20, 24), 2, False, 8), ("fcc", (17, 19, 18), 2, True, 12), ("fcc", (18, 18, 18), 2, False, 8),
    ("long", (520, 14, 13), 2, False, 12), ("long", (520, 13, 14), 1, True, 12)])
def test_force_and_stress(synth_psp8, kind, shape, ncol, kpt, order):
    from lynx_b200 import solver
    if kind == "fcc":
        cl, pos = C.fcc_si_primitive(shape[0])
        cl.shape = shape
    else:
        cl, pos = C.diamond_si(1, shape, displace=0.05, seed=4)
    cl.fd_order = order
    tab = P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8))
    t = dict(img_atom=tab.img_atom, img_ndc=tab.img_ndc, img_shift=tab.img_shift, img_coords=tab.img_coords,
             gpos=tab.gpos, chi=tab.chi, gamma=tab.gamma, nproj=int(tab.atom_nproj[0]), n_atom=tab.n_atom)
    ctx = solver.Context(cl)
    ctx.set_nonlocal(tab)
    k = np.array([0.15, -0.2, 0.3]) * 2 * np.pi / cl.lengths if kpt else None
    if kpt:
        ctx.set_kpoint(k)
    psi = C.random_orbitals(ctx.nd, ncol, seed=6, complex_=kpt)
    occ = np.linspace(1.0, 0.3, ncol)
    st = O.stencil(cl.latvec, cl.shape, order, cl.orthogonal)
    nl = solver.NonlocalProjector(ctx)
    f, e = nl.force(psi, occ, kpt=kpt)
    f_want, e_want = O.nonlocal_force(psi, occ, t, st, cl.shape, st["dV"], 2.0, 1.0, k, cl.lengths)
    assert np.abs(f - f_want).max() < 1e-11 * np.abs(f_want).max()
    assert abs(e - e_want) < 1e-11 * abs(e_want)
    sk, snl = nl.stress(psi, occ, kpt=kpt)
    sk_want, snl_want, _ = O.kinetic_nonlocal_stress(psi, occ, t, st, cl, st["dV"], 2.0, 1.0, k)
    assert np.abs(sk - sk_want).max() < 1e-11 * np.abs(sk_want).max()
    assert np.abs(snl - snl_want).max() < 1e-11 * np.abs(snl_want).max()
    ctx.close()
