"""Device memory of the velocity pipeline: enforcement after advection and redistancing on the same context takes next to
nothing more (its lists use the scratch of those calls, 12 bytes a cell otherwise)."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_enforcement_shares_scratch(sfpkg):
    import torch
    shape = (128, 128, 128)
    g = sfpkg.StaggeredGrid.from_origin(1 / 128, shape)
    ctx = sfpkg.Context(0)
    zeros = [torch.zeros(g.face_shape(a), dtype=torch.float64, device="cuda") for a in range(3)]
    frac = [torch.ones_like(z) for z in zeros]
    phi = torch.full(shape, -0.5, dtype=torch.float64, device="cuda")
    sfpkg.Advection(g, ctx).solve_velocity(zeros, 0.01, device=True)
    sfpkg.Reinitialization(g, ctx).solve(phi, 1, device=True)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    sfpkg.ColliderEnforce(g, frac, zeros, ctx=ctx).enforce(zeros, device=True)
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    sfpkg.Reinitialization(g, ctx).solve(phi, 1, device=True)  # and the scratch is as good as before
    assert np.isfinite(phi.cpu().numpy()).all()
    ctx.close()
    assert taken <= 4 * np.prod(shape), taken
