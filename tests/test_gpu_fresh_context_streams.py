"""First passes on contexts that no call has used yet, on streams that the legacy stream does not
order: the projector tables that a context lays out on first use must have arrived before the
kernels that read them.  Grids whose FP32 rows are padded (26, 30) and not (24, 28), so that both
kinds of table are made inside the call; results bitwise those of the same contexts afterwards."""
import numpy as np
import pytest

from lynx_b200 import _lib
from lynx_b200 import ensemble as E
from lynx_b200 import pseudo as P
from lynx_b200 import cell as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("trial", range(3))
def test_first_pass_in_a_batch(synth_psp8, precision, trial):
    from lynx_b200 import solver
    probs = E.strained_ensemble(P.read_psp8(synth_psp8), n_cells=6, grids=(24, 26, 28, 30), nband=16, seed=40 + trial)
    solvers, bounds = [], []
    for pb in probs:
        ctx = solver.Context(pb.cell)
        ctx.set_option(_lib.OPT_AUTOTUNE, 0)
        ctx.set_nonlocal(pb.tables)
        solvers.append(solver.EigenSolver(ctx, precision))
        lo, hi = float(pb.veff.min()) - 1.0, ctx.max_eigval_half_lap + 8.0
        bounds.append((0.5 * (lo + hi), lo, hi))
    psi = [C.random_orbitals(p.cell.nd, p.nband, seed=7 + i) for i, p in enumerate(probs)]
    got = solver.solve_batch(solvers, psi, [p.veff for p in probs], *[list(b) for b in zip(*bounds)], 6)
    for es, p, x, b, (y, eig) in zip(solvers, probs, psi, bounds, got):
        y1, eig1 = es.solve(x, p.veff, *b, 6)
        assert np.array_equal(eig, eig1)
        assert np.array_equal(y, y1)
