"""The jump kernel's rows (four faces a lane, one launch for the three axes) against the oracle bit for bit: rows that end
around the 128 faces of a pass, edge grids without edges, missing terms, densities that divide inexactly."""
import numpy as np
import pytest

from conftest import oracle_grid


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 127), (3, 2, 128), (2, 9, 129), (1, 3, 31), (4, 17, 260)])
@pytest.mark.parametrize("terms", ["both", "kappa", "pm", "none"])
def test_jump_rows_vs_oracle(sfpkg, oracle, gpu_ctx, shape, terms):
    rng = np.random.default_rng(sum(shape))
    g = sfpkg.StaggeredGrid.from_origin(0.3, shape)
    nv = 50
    marks = [np.where(rng.random(tuple(s - (a == b) for b, s in enumerate(shape))) < 0.4, rng.integers(0, nv, 1), -1)
             .astype(np.int32) for a in range(3)]
    kappa = rng.standard_normal(nv) if terms in ("both", "kappa") else None
    pm = rng.standard_normal(nv) * 1e-320 if terms == "pm" else (rng.standard_normal(nv) if terms == "both" else None)
    want = oracle.pressure_jump(oracle_grid(oracle, g), marks, kappa, pm, 0.07, 1.3, 0.01)
    got = sfpkg.pressure_jump(g, marks, kappa, pm, 0.07, 1.3, 0.01, ctx=gpu_ctx)
    for a in range(3):
        assert np.array_equal(got[a], want[a])
