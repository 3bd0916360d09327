"""Expansion tiles whose alpha rows come close to the default shared-memory limit (21 atoms in a tile at
this density), and around it: the fused nonlocal term bitwise the separate one."""
import numpy as np
import pytest

from lynx_b200 import _lib
from lynx_b200 import cell as C
from lynx_b200 import pseudo as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(75, 75, 73), (72, 73, 74), (74, 76, 78), (84, 84, 84)])
def test_fused_term_of_many_atoms(synth_psp8, shape):
    from lynx_b200 import solver
    cl, pos = C.diamond_si(3, shape, displace=0.02, seed=2)
    V = C.synthetic_veff_separable(cl, pos)
    ctx = solver.Context(cl)
    ctx.set_option(_lib.OPT_AUTOTUNE, 0)
    ctx.set_nonlocal(P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8)))
    x = C.random_orbitals(ctx.nd, 2, seed=3)
    for precision in ("mixed", "fp64"):
        out = []
        for fuse in (1, 0):
            ctx.set_option(_lib.OPT_FUSE_NONLOCAL, fuse)
            out.append(solver.EigenSolver(ctx, precision).chebyshev_filter(x, V, 25.0, -2.0, 70.0, degree=2))
        assert np.array_equal(out[0], out[1])
    ctx.close()
