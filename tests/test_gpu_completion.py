"""Operator calls are complete when they return, whichever kernels they run and whatever the context ran
before: the work uses blocks of the context, and the next call may come on another stream.  One
context, two streams that nothing orders; results bitwise those of one stream."""
import numpy as np
import pytest

from helpers import si8_small
from lynx_b200 import cell as C
from lynx_b200 import pseudo as P

pytestmark = pytest.mark.gpu

LONG = 40_000_000  # clock cycles ahead of the call on its stream: above 20 ms


@pytest.fixture
def si8(synth_psp8):
    from lynx_b200 import solver
    cl, pos, V = si8_small(grid=(20, 21, 22))
    ctx = solver.Context(cl)
    ctx.set_nonlocal(P.nonlocal_tables(cl, pos, P.read_psp8(synth_psp8)))
    ctx.set_kpoint(np.array([0.25, -0.125, 0.375]) * 2 * np.pi / cl.lengths)
    yield cl, V, ctx
    ctx.close()


def _block(ctx, ncol, seed, kpt):
    import torch
    x = C.random_orbitals(ctx.nd, ncol, seed=seed, complex_=kpt)
    return torch.from_numpy(np.ascontiguousarray(x.T)).cuda()


def _call(ctx, what, kpt):
    from lynx_b200 import solver
    if what == "apply":
        h = solver.Hamiltonian(ctx)
        return lambda x, V: (h.apply_kpt if kpt else h.apply)(x, Veff=V)
    es = solver.EigenSolver(ctx, what)
    return lambda x, V: es.chebyshev_filter(x, V, 25.0, -2.0, 70.0, degree=6, kpt=kpt)


@pytest.mark.parametrize("what", ["apply", "fp64", "mixed"])
@pytest.mark.parametrize("kpt,ncol", [(True, 6), (False, 3), (False, 40)])
def test_complete_on_return_on_any_stream(si8, what, kpt, ncol):
    import torch
    cl, V, ctx = si8
    f = _call(ctx, what, kpt)
    V = torch.from_numpy(V).cuda()
    xs = [_block(ctx, ncol, 3 + i, kpt) for i in range(2)]
    want = [f(x, V).clone() for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = []
    for s, x in zip(streams, xs):
        with torch.cuda.stream(s):
            torch.cuda._sleep(LONG)
            got.append(f(x, V))
        assert s.query(), "the call returned with work in flight"
    for g, w in zip(got, want):
        assert torch.equal(g, w)


def test_recorded_call_replays(si8):
    """A call whose kernels have no bounded waits can be recorded after a first call."""
    import torch
    cl, V, ctx = si8
    f = _call(ctx, "apply", True)
    V = torch.from_numpy(V).cuda()
    x = _block(ctx, 4, 5, True)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        want = f(x, V).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        y = f(x, V)
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


@pytest.mark.parametrize("kpt", [False, True])
def test_nonlocal_apply_on_another_stream_waits(si8, kpt):
    """The nonlocal apply returns with its work in flight; one on another stream, which uses the same
    projections of the context, waits for it."""
    import time
    import torch
    from lynx_b200 import solver
    cl, V, ctx = si8
    nl = solver.NonlocalProjector(ctx)
    xs = [_block(ctx, 5, 3 + i, kpt) for i in range(2)]
    want = [nl.apply(x, torch.zeros_like(x), kpt=kpt).clone() for x in xs]
    got = [torch.zeros_like(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(20 * LONG)
        nl.apply(xs[0], got[0], kpt=kpt)
    with torch.cuda.stream(streams[1]):
        nl.apply(xs[1], got[1], kpt=kpt)
    time.sleep(0.05)
    assert not streams[0].query() and not streams[1].query()
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert torch.equal(g, w)
