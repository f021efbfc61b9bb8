"""The ghost-element copies of the time loop and the zero ghosts of a right-hand side against whole-
state copies: every ghost value exactly, every interior value untouched."""
import numpy as np
import pytest
import torch

from helpers import INNER

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("res,n", [((1, 1, 1), 2), ((2, 1, 3), 3), ((3, 2, 1), 5), ((2, 33, 50), 8), ((1, 4, 5), 10)])
def test_ghost_elements(cuda, res, n, precision):
    from vlasov1d2v_b200 import problem
    from vlasov1d2v_b200.context import get_context

    p = problem.build(res, n, perturbation=None, precision=precision, background_split=False)
    ctx = get_context(p.grids, precision=precision)
    dt = torch.float64 if precision == "fp64" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n)
    f, sa, sb, out = (torch.rand(ctx.state_shape, dtype=dt, device="cuda", generator=g) for _ in range(4))
    want_f = f.clone()
    want_f[0], want_f[-1] = f[-2], f[1]
    ghost = torch.ones(ctx.state_shape, dtype=torch.bool, device="cuda")
    ghost[INNER] = False
    velocity_ghost = ghost.clone()
    velocity_ghost[0] = velocity_ghost[-1] = False
    want = [torch.where(velocity_ghost, f, s) for s in (sa, sb)]
    ctx.sync_stage_ghosts(f, sa, sb)
    E = torch.zeros((res[0] + 2, n), dtype=torch.float64, device="cuda")
    interior = torch.zeros_like(out)
    ctx.rhs(f, E, interior)
    want_out = torch.where(ghost, torch.zeros_like(out), interior)
    ctx.rhs_whole(f, E, out)
    assert torch.equal(f, want_f)
    assert torch.equal(sa, want[0]) and torch.equal(sb, want[1])
    assert torch.equal(out, want_out)


def test_rhs_ghosts_are_zero(cuda):
    """``DGFlux.semi_discrete_rhs`` into uninitialised memory: zero ghost elements."""
    from vlasov1d2v_b200 import problem

    p = problem.build((2, 3, 4), 4, perturbation="cos", amp=0.1)
    junk = [torch.full(tuple(p.f.arr.shape), float("nan"), dtype=torch.float64, device="cuda") for _ in range(3)]
    del junk   # the allocator hands this memory out again
    r = p.flux.semi_discrete_rhs(p.f.arr, p.elliptic, p.basis, p.grids).get()
    assert np.isfinite(r).all()
    r[INNER] = 0.0
    assert not r.any()
