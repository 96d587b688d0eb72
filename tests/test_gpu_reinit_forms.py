"""The redistancing kernel's two forms (integer-pipe and plain FP64) and its skipped one-sided derivatives, against the
oracle bit for bit: grids shorter than the stencil, plane fields (exact zero differences on two axes), fields whose
differences leave the fast form's range, kinks, infinities and NaN."""
import numpy as np
import pytest

from conftest import oracle_grid


def _field(kind, g, rng):
    s = g.shape
    c = [(np.arange(s[a]) + 0.5) * g.spacing for a in range(3)]
    X, Y, Z = np.meshgrid(*c, indexing="ij")
    if kind == "plane":
        return Y - 0.37
    if kind == "noise":
        return rng.standard_normal(s)
    if kind == "kinks":
        return np.abs(np.sin(9 * X)) - np.abs(Y - 0.3) + np.round(Z * 3)
    if kind == "steps":  # zero and nonzero differences mixed, an exactly zero level set on part of the grid
        return np.floor(4 * X) * 0.25 - np.floor(3 * Z) * 0.5
    if kind == "tiny":
        return rng.standard_normal(s) * 1e-200
    if kind == "huge":
        return rng.standard_normal(s) * 1e100
    if kind == "spread":  # magnitudes over the fast form's range and beyond
        return rng.standard_normal(s) * 2.0 ** rng.integers(-140, 80, s)
    f = rng.standard_normal(s)
    f[tuple(n // 2 for n in s)] = np.inf if kind == "inf" else np.nan
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plane", "noise", "kinks", "steps", "tiny", "huge", "spread", "inf", "nan"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 5, 3), (7, 9, 33), (20, 12, 70)])
def test_reinitialize_forms_vs_oracle(sfpkg, oracle, gpu_ctx, kind, shape):
    g = sfpkg.StaggeredGrid.from_origin(1.0 / 13, shape)
    phi = np.ascontiguousarray(_field(kind, g, np.random.default_rng(sum(shape))))
    with np.errstate(all="ignore"):
        want = oracle.reinitialize(oracle_grid(oracle, g), phi, 2)
    got = phi.copy()
    sfpkg.Reinitialization(g, gpu_ctx).solve(got, 2)
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("h", [1e-25, 0.1, 1e25])
def test_reinitialize_spacings_vs_oracle(sfpkg, oracle, gpu_ctx, h):
    """Spacings beyond the fast form's range take the plain one."""
    g = sfpkg.StaggeredGrid.from_origin(h, (9, 8, 34))
    phi = np.ascontiguousarray(_field("noise", g, np.random.default_rng(3)) * h)
    got = phi.copy()
    sfpkg.Reinitialization(g, gpu_ctx).solve(got, 2)
    assert np.array_equal(got, oracle.reinitialize(oracle_grid(oracle, g), phi, 2))
