"""Advection's two forms (integer-pipe and plain FP64), its shortcuts for still air and for points that sit on cells, and
its table of first points, against the oracle bit for bit: spacings that are powers of two and not, grids narrower than
the stencil, velocities that are zero, along one axis, large and tiny, and level sets outside the integer form's range.
(Infinite velocities are left out: a departure point at infinity has no integer cell in C.)"""
import numpy as np
import pytest

from conftest import oracle_grid


def _velocity(kind, faces, h, rng):
    u = [rng.uniform(-1, 1, f) for f in faces]
    if kind == "still":
        return [np.zeros(f) for f in faces]
    if kind == "half":  # still beyond half of the domain, as the extrapolation leaves it
        return [np.where(np.arange(f[1])[None, :, None] < f[1] // 2, a, 0.0) for a, f in zip(u, faces)]
    if kind == "axis":  # motion along y by whole cells: the other axes' weights stay 0, 1, 0, 0
        return [np.zeros(faces[0]), np.full(faces[1], 1.0), np.zeros(faces[2])]
    if kind == "fast":
        return [a * 40 for a in u]
    if kind == "tiny":
        return [a * 1e-130 for a in u]
    if kind == "wide":
        return [a * 2.0 ** rng.integers(-400, 3, a.shape) for a in u]
    raise KeyError(kind)


def _level(kind, shape, rng):
    phi = rng.uniform(-1, 1, shape)
    if kind == "zeros":
        return phi * (rng.random(shape) < 0.5)
    if kind == "wide":
        return phi * 2.0 ** rng.integers(-180, 350, shape)
    if kind == "inf":
        phi.flat[phi.size // 2] = np.inf
    return phi


@pytest.mark.gpu
@pytest.mark.parametrize("h", [1 / 16, 0.07])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 5), (6, 9, 33), (12, 10, 40)])
@pytest.mark.parametrize("vel,level", [("still", "plain"), ("still", "zeros"), ("still", "inf"), ("half", "plain"),
                                       ("half", "wide"), ("axis", "plain"), ("axis", "inf"), ("fast", "plain"),
                                       ("tiny", "zeros"), ("wide", "plain")])
def test_advection_forms_vs_oracle(sfpkg, oracle, gpu_ctx, h, shape, vel, level):
    rng = np.random.default_rng(sum(shape) + len(vel))
    g = sfpkg.StaggeredGrid.from_origin(h, shape)
    og = oracle_grid(oracle, g)
    u = _velocity(vel, [g.face_shape(a) for a in range(3)], h, rng)
    phi = np.ascontiguousarray(_level(level, shape, rng))
    u = [np.ascontiguousarray(a) for a in u]
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
