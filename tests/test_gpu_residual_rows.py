"""The mixed form's FP64 residual by rows of one exact coupling: the residuals that the solver reports against b - A x
formed here from the operator and right-hand side that it read back.

Tolerance, before the first run: the integer sum drops less than 2^-58 max|x| of each of a row's seven values (scaled by the
coupling, at most 1 + chi), at most 12 (1 + chi) 2^-58 max|x| a cell; the FP64 evaluation here errs by about 8 eps
(1 + chi) 6 max|x| a cell.  Both over n cells and ||b||, twice their sum."""
import numpy as np
import pytest

from conftest import scenes


def _residual(diag, lower, b, x):
    r = b - diag * x
    for a in range(3):
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[a], hi[a] = slice(0, -1), slice(1, None)
        lo, hi = tuple(lo), tuple(hi)
        r[hi] += lower[a][hi] * x[lo]
        r[lo] += lower[a][hi] * x[hi]
    return r


def _bound(b, x, c):
    return 2 * np.sqrt(b.size) * c * np.abs(x).max() * (12 * 2.0 ** -58 + 48 * 2.0 ** -53) / np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(9, 7, 8), (17, 20, 72), (8, 33, 64), (40, 24, 136)])
@pytest.mark.parametrize("chi", [0.7, 2.0])
def test_reported_potential_residual(sfpkg, gpu_ctx, shape, chi):
    g = sfpkg.StaggeredGrid.from_origin(1 / 16, shape)
    rng = np.random.default_rng(sum(shape))
    y = scenes().cell_centres(g, 1)
    phi = np.ascontiguousarray(np.broadcast_to((y - 0.4 * y.max())[None, :, None], shape)) + 1e-3 * rng.random(shape)
    hext = [np.ascontiguousarray(rng.standard_normal(g.face_shape(a))) for a in range(3)]
    M = sfpkg.MagneticField(g, chi, 2 * g.spacing, gpu_ctx)
    for tol in (1e-4, 1e-7, 1e-9):  # the later ones start from the last potential
        st = M.solve(phi, hext, opts=sfpkg.options("magnetic", precision="mixed", tol=tol))
        diag, lower, b = gpu_ctx.system_operator(1, shape)
        r = _residual(diag, lower, b, M.potential)
        tolerance = _bound(b, M.potential, 1 + chi)
        r[0, 0, 0] = b[0, 0, 0] = 0.0  # the pinned row
        got, want = st["rel_residual_ref"], np.linalg.norm(r) / np.linalg.norm(b)
        assert abs(got - want) <= tolerance + 1e-12 * want, (got, want, tolerance)
        assert st["rel_residual"] <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(12, 9, 8), (24, 40, 72)])
def test_reported_pressure_residual(sfpkg, gpu_ctx, shape):
    g = sfpkg.StaggeredGrid.from_origin(1 / 16, shape)
    rng = np.random.default_rng(sum(shape))
    y = scenes().cell_centres(g, 1)
    phi = np.ascontiguousarray(np.broadcast_to((y - 0.6 * y.max())[None, :, None], shape)) + 1e-3 * rng.random(shape)
    frac = [np.ascontiguousarray(rng.choice([0.0] * 200 + [0.25, 1.0], g.face_shape(a))) for a in range(3)]
    P = sfpkg.Pressure(g, gpu_ctx)
    for call in (P.project, P.reproject):
        u = [rng.standard_normal(g.face_shape(a)) for a in range(3)]
        st = call(u, phi, frac, opts=sfpkg.options("pressure", precision="mixed", tol=1e-9))
        diag, lower, b = gpu_ctx.system_operator(0, shape)
        r = _residual(diag, lower, b, P.pressure)
        want = np.linalg.norm(r) / np.linalg.norm(b)
        assert abs(st["rel_residual"] - want) <= _bound(b, P.pressure, diag.max() / 6) + 1e-12 * want
