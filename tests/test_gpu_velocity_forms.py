"""Extrapolation by validity bits and enforcement by face lists, against the oracle bit for bit: rows that end at, before
and after a 32-bit word, every number of sweeps, solid faces inside the domain and on all of it, moving solids, and
velocities that are zero or infinite where the interpolation reads them."""
import numpy as np
import pytest

from conftest import oracle_grid


def _case(shape, seed, solid):
    rng = np.random.default_rng(seed)
    phi = rng.uniform(-1, 1, shape) - 0.3 if solid != "dry" else np.ones(shape)
    faces = [tuple(s + (a == b) for b, s in enumerate(shape)) for a in range(3)]
    frac = [np.where(rng.random(f) < 0.3, 1.0, rng.choice([0.0, 0.4], f)) for f in faces]
    if solid == "all":
        frac = [np.ones(f) for f in faces]
    elif solid == "none":
        frac = [np.zeros(f) for f in faces]
    u = [rng.uniform(-1, 1, f) * (rng.random(f) < 0.7) for f in faces]
    normal = [rng.uniform(-1, 1, f) * (rng.random(f) < 0.5) for f in faces]
    return phi, frac, u, normal, rng


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 31), (2, 3, 32), (5, 4, 33), (4, 40, 63), (9, 7, 64), (6, 70, 65)])
@pytest.mark.parametrize("solid", ["some", "all", "none", "dry"])
def test_extrapolation_by_bits_vs_oracle(sfpkg, oracle, gpu_ctx, shape, solid):
    g = sfpkg.StaggeredGrid.from_origin(1.0 / shape[0], shape)
    phi, frac, u, _, _ = _case(shape, sum(shape), solid)
    for steps, clear in ((0, 0.0), (1, 0.25), (2, 0.0), (7, -1.5)):
        want = oracle.extrapolate_velocity(oracle_grid(oracle, g), u, phi, frac, clear, steps)
        v = [a.copy() for a in u]
        sfpkg.Extrapolation(g, gpu_ctx).solve(v, phi, frac, clear, steps)
        for a in range(3):
            assert np.array_equal(v[a], want[a]), (steps, a)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 31), (5, 4, 33), (20, 21, 40)])
@pytest.mark.parametrize("solid", ["some", "all", "none"])
@pytest.mark.parametrize("moving", [False, True])
def test_enforcement_by_lists_vs_oracle(sfpkg, oracle, gpu_ctx, shape, solid, moving):
    g = sfpkg.StaggeredGrid.from_origin(1.0 / 7, shape)
    _, frac, u, normal, rng = _case(shape, sum(shape) + 1, solid)
    us = [rng.uniform(-1, 1, a.shape) for a in u] if moving else None
    if moving:
        u[0].flat[u[0].size // 2] = np.inf  # beside zeros: 0 inf is NaN
    with np.errstate(all="ignore"):
        want = oracle.collider_enforce(oracle_grid(oracle, g), u, frac, normal, us)
    v = [a.copy() for a in u]
    sfpkg.ColliderEnforce(g, frac, normal, us, ctx=gpu_ctx).enforce(v)
    for a in range(3):
        assert np.array_equal(v[a], want[a], equal_nan=True), a
