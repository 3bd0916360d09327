"""lynx_pair_density (the potential's gradient of H psi): even and odd point counts, an unaligned block,
one and many columns; and second derivatives still go through torch when the backward is recorded, as
do backwards of many gradients at once."""
import numpy as np
import pytest

from lynx_b200 import cell as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,ncol", [((16, 17, 18), 1), ((17, 15, 19), 5), ((16, 16, 16), 33)])
@pytest.mark.parametrize("shift", [0, 1])
def test_pair_density(shape, ncol, shift):
    import torch
    from lynx_b200 import solver
    ctx = solver.Context(C.diamond_si(1, shape)[0])
    g = torch.Generator(device="cuda").manual_seed(1)
    buf = [torch.rand(ncol * ctx.nd + 1, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    u, v = [b[shift:shift + ncol * ctx.nd].view(ncol, ctx.nd) for b in buf]
    out = solver.pair_density(ctx, u, v)
    want = (u * v).sum(0)
    assert float((out - want).abs().max()) <= 2 * ncol * 2.0 ** -53 * float(want.abs().max())
    ctx.close()


def test_recorded_backward_stays_differentiable():
    import torch
    from lynx_b200 import autograd, solver
    ctx = solver.Context(C.diamond_si(1, (16, 16, 16))[0])
    psi = torch.rand(2, ctx.nd, dtype=torch.float64, device="cuda", requires_grad=True)
    veff = torch.rand(ctx.nd, dtype=torch.float64, device="cuda", requires_grad=True)
    g = torch.rand(2, ctx.nd, dtype=torch.float64, device="cuda")
    y = autograd.hamiltonian_apply(ctx, psi, veff)
    (gv,) = torch.autograd.grad(y, veff, g, create_graph=True)
    (gp,) = torch.autograd.grad(gv.sum(), psi)
    assert np.allclose(gp.cpu().numpy(), g.cpu().numpy())
    ctx.close()


def test_batched_backward_in_the_potential():
    """is_grads_batched runs the backward under vmap, whose tensors have no memory to point at."""
    import torch
    from lynx_b200 import autograd, solver
    ctx = solver.Context(C.diamond_si(1, (16, 16, 16))[0])
    psi = torch.rand(2, ctx.nd, dtype=torch.float64, device="cuda")
    veff = torch.rand(ctx.nd, dtype=torch.float64, device="cuda", requires_grad=True)
    g = torch.rand(3, 2, ctx.nd, dtype=torch.float64, device="cuda")
    y = autograd.hamiltonian_apply(ctx, psi, veff)
    (gv,) = torch.autograd.grad(y, veff, g, is_grads_batched=True)
    want = (g * psi).sum(1)
    assert float((gv - want).abs().max()) <= 2 ** -51 * float(want.abs().max())
    ctx.close()
