"""Grids so long in y that a launch with a block row for every four rows of y leaves the launch limits (65,535 blocks), and
grids as long in z and x as the other kernels take: the redistancing against the oracle bit for bit."""
import numpy as np
import pytest

from conftest import oracle_grid


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 262145, 3), (1, 300000, 2), (2, 3, 200001), (65535, 2, 3)])
def test_reinitialize_long(sfpkg, oracle, gpu_ctx, shape):
    g = sfpkg.StaggeredGrid.from_origin(1 / 8, shape)
    rng = np.random.default_rng(3)
    s = np.indices(shape).sum(axis=0) % 64
    phi = np.ascontiguousarray((s - 31.3) / 8 + 0.01 * rng.standard_normal(shape))
    want = oracle.reinitialize(oracle_grid(oracle, g), phi, 1)
    got = phi.copy()
    sfpkg.Reinitialization(g, gpu_ctx).solve(got, 1)
    assert np.array_equal(got, want)
