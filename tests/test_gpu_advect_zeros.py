"""Advection of and by fields with exact zeros, infinities and tiny values among ordinary ones, where one sample mixes the
integer form with rows or points in FP64: against the oracle bit for bit, on moving points."""
import numpy as np
import pytest

from conftest import oracle_grid


def _level(kind, shape, rng):
    phi = rng.uniform(-1, 1, shape)
    if kind == "scattered":
        return phi * (rng.random(shape) < 0.5)
    if kind == "layer":  # the surface passes through a layer of cells
        phi[:, shape[1] // 2, :] = -0.0
    if kind == "tiny":
        return np.where(rng.random(shape) < 0.3, phi * 2.0 ** rng.integers(-1070, -90, shape), phi)
    if kind == "inf":
        phi.flat[rng.integers(0, phi.size, 1 + phi.size // 50)] = np.inf
        phi.flat[rng.integers(0, phi.size, 1 + phi.size // 50)] = np.nan
    return phi


@pytest.mark.gpu
@pytest.mark.parametrize("h", [1 / 16, 0.07])
@pytest.mark.parametrize("shape", [(3, 2, 5), (6, 9, 33), (12, 10, 40)])
@pytest.mark.parametrize("vel", ["all", "one axis", "some zero"])
@pytest.mark.parametrize("level", ["scattered", "layer", "tiny", "inf"])
def test_advection_with_zeros_vs_oracle(sfpkg, oracle, gpu_ctx, h, shape, vel, level):
    rng = np.random.default_rng(sum(shape) + len(vel) + len(level))
    g = sfpkg.StaggeredGrid.from_origin(h, shape)
    og = oracle_grid(oracle, g)
    u = [rng.uniform(-1.5, 1.5, g.face_shape(a)) for a in range(3)]
    if vel == "one axis":
        u[0][:] = 0.0
        u[2][:] = 0.0
    if vel == "some zero":
        u = [a * (rng.random(a.shape) < 0.7) for a in u]
    phi = np.ascontiguousarray(_level(level, shape, rng))
    with np.errstate(all="ignore"):
        want = oracle.advect_levelset(og, phi, u, h)
        want_u = oracle.advect_velocity(og, u, h)
    got = phi.copy()
    sfpkg.Advection(g, gpu_ctx).solve_levelset(got, u, h)
    assert np.array_equal(got, want, equal_nan=True)
    v = [a.copy() for a in u]
    sfpkg.Advection(g, gpu_ctx).solve_velocity(v, h)
    for a in range(3):
        assert np.array_equal(v[a], want_u[a], equal_nan=True)
