"""The coarsest solve on grids of odd and even rows, one cell thick and of the most cells it takes in one block: one
preconditioned step of a one-level hierarchy from zero against the same sweeps formed here from the operator and
right-hand side that the solver reads back.

Tolerance, before the first run: 97 half sweeps of sums of eight terms in another rounding (the kernel contracts
a x + s), each contracting the error it is given: 97 x 8 eps = 1.7e-13 of max|p|, the step length's two sums of up to 1024
terms as much again; ten times that."""
import numpy as np
import pytest


def _matvec(diag, lower, x):
    s = np.zeros_like(x)
    for a in range(3):
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[a], hi[a] = slice(0, -1), slice(1, None)
        lo, hi = tuple(lo), tuple(hi)
        s[hi] += lower[a][hi] * x[lo]
        s[lo] += lower[a][hi] * x[hi]
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("closed", [False, True])
@pytest.mark.parametrize("shape", [(8, 8, 8), (5, 4, 4), (9, 7, 9), (3, 5, 67), (32, 32, 1), (2, 512, 1), (1, 1, 1024)])
def test_one_step(sfpkg, gpu_ctx, shape, closed):
    g = sfpkg.StaggeredGrid.from_origin(1 / 16, shape)
    rng = np.random.default_rng(sum(shape))
    phi = np.full(shape, -1.0) if closed else np.ascontiguousarray(rng.uniform(-1, 0.2, shape))
    frac = [np.zeros(g.face_shape(a)) for a in range(3)]
    u = [rng.standard_normal(g.face_shape(a)) for a in range(3)]
    P = sfpkg.Pressure(g, gpu_ctx)
    P.project(u, phi, frac, opts=sfpkg.options("pressure", precision="fp64", max_levels=1, max_iters=1, coarse_sweeps=48,
                                               warm_start=0), raise_on_nonconv=False)
    diag, lower, b = gpu_ctx.system_operator(0, shape)
    act = diag > 0
    inv = np.where(act, 1 / np.where(act, diag, 1), 0)
    r = b.copy()
    if np.abs(diag - _matvec(diag, lower, np.ones(shape))).max() <= 1e-9 * diag.max():
        r = np.where(act, r - r[act].mean(), r)
    colour = np.add.outer(np.add.outer(np.arange(shape[0]), np.arange(shape[1])), np.arange(shape[2])) & 1
    z = np.zeros(shape)
    for h in range(97):
        z = np.where(colour == (h & 1), (r + _matvec(diag, lower, z)) * inv, z)
    az = diag * z - _matvec(diag, lower, z)
    want = (b * z).sum() / (z * az).sum() * z
    assert np.abs(P.pressure - want).max() <= 10 * 2 * 97 * 8 * 2.0 ** -52 * np.abs(want).max()
