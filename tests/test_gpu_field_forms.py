"""The total field's forms (1 / h a power of two or not, potentials inside and outside the integer product's range) and
the projection's face order, against the oracle: the field bit for bit from the library's own potential, the velocity
bit for bit from the library's own pressure, with partly open, closed and surface faces and a jump."""
import numpy as np
import pytest

from conftest import oracle_grid


@pytest.mark.gpu
@pytest.mark.parametrize("h", [1 / 16, 0.07])
@pytest.mark.parametrize("scale", [1.0, 1e-170, 1e170])
@pytest.mark.parametrize("shape", [(5, 3, 4), (16, 12, 33), (20, 16, 40)])
def test_total_field_forms(sfpkg, gpu_ctx, h, scale, shape):
    rng = np.random.default_rng(sum(shape))
    g = sfpkg.StaggeredGrid.from_origin(h, shape)
    phi = np.ascontiguousarray(rng.uniform(-1, 1, shape))
    hext = [np.ascontiguousarray(rng.standard_normal(g.face_shape(a)) * scale) for a in range(3)]
    hext[1].flat[3] = -0.0
    M = sfpkg.MagneticField(g, 1.5, 2 * h, gpu_ctx)
    M.solve(phi, hext, opts=sfpkg.options("magnetic", max_iters=3, warm_start=0), raise_on_nonconv=False)
    psi, invh = M.potential, 1 / h
    for a in range(3):
        want = hext[a] + 0.0
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[a], hi[a] = slice(0, -1), slice(1, None)
        mid = [slice(None)] * 3
        mid[a] = slice(1, -1)
        with np.errstate(all="ignore"):
            want[tuple(mid)] = (psi[tuple(lo)] - psi[tuple(hi)]) * invh + hext[a][tuple(mid)]
        assert np.array_equal(M.total_field[a], want, equal_nan=True), a


@pytest.mark.gpu
@pytest.mark.parametrize("jump", [False, True])
@pytest.mark.parametrize("shape", [(3, 4, 5), (12, 10, 33), (16, 20, 40)])
def test_projection_faces(sfpkg, gpu_ctx, jump, shape):
    rng = np.random.default_rng(sum(shape) + jump)
    g = sfpkg.StaggeredGrid.from_origin(1 / 16, shape)
    phi = np.ascontiguousarray(rng.uniform(-1, 0.6, shape))
    faces = [g.face_shape(a) for a in range(3)]
    frac = [np.ascontiguousarray(rng.choice([0.0, 0.0, 0.3, 1.0], f)) for f in faces]
    u = [rng.standard_normal(f) for f in faces]
    J = [np.ascontiguousarray(rng.standard_normal(f)) for f in faces] if jump else None
    P = sfpkg.Pressure(g, gpu_ctx)
    P.set_pressure_jump(J)
    v = [a.copy() for a in u]
    P.project(v, phi, frac, raise_on_nonconv=False)
    p, liq = P.pressure, phi <= 0
    for a in range(3):
        want = u[a].copy()
        n = shape[a]
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[a], hi[a] = slice(0, n - 1), slice(1, n)
        lo, hi = tuple(lo), tuple(hi)
        mid = tuple(slice(1, n) if b == a else slice(None) for b in range(3))
        w, l0, l1 = 1 - frac[a][mid], liq[lo], liq[hi]
        pj = J[a][mid] if jump else 0.0
        with np.errstate(all="ignore"):
            theta = phi[lo] / (phi[lo] - phi[hi])
            t = np.where(l0, theta, 1 - theta)
            ic = 1.0 / np.where(t < 0.001, 0.001, t)
            one = np.where(l0, 1.0, -1.0) * (pj - np.where(l0, p[lo], p[hi])) * ic * w
            du = np.where(l0 & l1, (p[hi] - p[lo]) * w, one)
        want[mid] = np.where((w > 0) & (l0 | l1), want[mid] - du, want[mid])
        assert np.array_equal(v[a], want), a
