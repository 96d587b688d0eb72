"""The total field at spacings far from one, against (psi - psi') / h + Hext bit for bit from the library's own potential:
1 / h inside and outside the integer product's range, with products that are normal, subnormal and infinite."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("h,scale", [(1e160, 1e-309), (1e-160, 2e307), (1e125, 1e-270), (1e-118, 1.0), (2.0 ** 450, 1e-290),
                                     (2.0 ** -450, 1e270), (3.0, 1.0)])
@pytest.mark.parametrize("shape", [(5, 3, 4), (9, 8, 33)])
def test_total_field_spacings(sfpkg, gpu_ctx, h, scale, shape):
    rng = np.random.default_rng(sum(shape))
    g = sfpkg.StaggeredGrid.from_origin(h, shape)
    phi = np.ascontiguousarray(rng.uniform(-1, 1, shape) * h)
    hext = [np.ascontiguousarray(rng.standard_normal(g.face_shape(a)) * scale) for a in range(3)]
    M = sfpkg.MagneticField(g, 1.5, 2 * h, gpu_ctx)
    M.solve(phi, hext, opts=sfpkg.options("magnetic", max_iters=3, warm_start=0), raise_on_nonconv=False)
    psi, invh = M.potential, 1 / h
    assert np.abs(psi).max() > 0  # the right-hand side did not leave the range of doubles
    for a in range(3):
        want = hext[a] + 0.0
        lo, hi, mid = ([slice(None)] * 3 for _ in range(3))
        lo[a], hi[a], mid[a] = slice(0, -1), slice(1, None), slice(1, -1)
        with np.errstate(all="ignore"):
            want[tuple(mid)] = (psi[tuple(lo)] - psi[tuple(hi)]) * invh + hext[a][tuple(mid)]
        assert np.array_equal(M.total_field[a], want, equal_nan=True), a
