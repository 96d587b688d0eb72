"""The mixed form's FP64 residual on either side of the rule that picks its kernel (three 64 x 8 x 8 items an SM): the
residuals that the solver reports against b - A x formed here from the operator and right-hand side that it read back.

Tolerance, before the first run: the integer sum drops less than 6 2^-58 max|x| a cell (times the coupling, at most 1 + chi),
its D is off by less than 18 2^-53 (1 + chi); the FP64 evaluations err by about 8 eps (1 + chi) 6 max|x| a cell.  Over n
cells and ||b||, twice their sum."""
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


# items: 460 and 504 (ragged in x and y), 468 (ragged in z and y); 440: below the rule
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(160, 184, 8), (161, 185, 8), (100, 140, 72), (160, 176, 8)])
@pytest.mark.parametrize("chi", [0.7, 2.0])
def test_reported_potential_residual(sfpkg, gpu_ctx, shape, chi):
    g = sfpkg.StaggeredGrid.from_origin(1 / 64, shape)
    rng = np.random.default_rng(sum(shape))
    y = scenes().cell_centres(g, 1)
    phi = np.ascontiguousarray(np.broadcast_to((y - 0.4 * y.max())[None, :, None], shape)) + 1e-3 * rng.random(shape)
    hext = [np.ascontiguousarray(rng.standard_normal(g.face_shape(a))) for a in range(3)]
    M = sfpkg.MagneticField(g, chi, 2 * g.spacing, gpu_ctx)
    for tol in (1e-4, 1e-9):  # the later one starts from the last potential
        st = M.solve(phi, hext, opts=sfpkg.options("magnetic", precision="mixed", tol=tol))
        diag, lower, b = gpu_ctx.system_operator(1, shape)
        x = M.potential
        r = _residual(diag, lower, b, x)
        bound = 2 * np.sqrt(b.size) * (1 + chi) * np.abs(x).max() * (6 * 2.0 ** -58 + (18 + 48) * 2.0 ** -53)
        bound /= np.linalg.norm(b)
        r[0, 0, 0] = b[0, 0, 0] = 0.0  # the pinned row
        got, want = st["rel_residual_ref"], np.linalg.norm(r) / np.linalg.norm(b)
        assert abs(got - want) <= bound + 1e-12 * want, (got, want, bound)
        assert st["rel_residual"] <= tol
