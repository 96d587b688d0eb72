"""The jump kernel's gathers (four faces a lane, passes of 128 faces): every marked edge with an index of its own draw, so that
a mark, curvature or pressure taken for another face shows, against the oracle bit for bit."""
import numpy as np
import pytest

from conftest import oracle_grid


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 1, 127), (3, 2, 128), (2, 9, 129), (4, 17, 260), (9, 8, 7)])
@pytest.mark.parametrize("share", [0.4, 1.0])
def test_jump_marks_vs_oracle(sfpkg, oracle, gpu_ctx, shape, share):
    rng = np.random.default_rng(sum(shape))
    g = sfpkg.StaggeredGrid.from_origin(0.3, shape)
    nv = 1000
    edges = [tuple(s - (a == b) for b, s in enumerate(shape)) for a in range(3)]
    marks = [np.where(rng.random(e) < share, rng.integers(0, nv, e), -1).astype(np.int32) for e in edges]
    kappa, pm = rng.standard_normal(nv), rng.standard_normal(nv)
    want = oracle.pressure_jump(oracle_grid(oracle, g), marks, kappa, pm, 0.07, 1.3, 0.01)
    got = sfpkg.pressure_jump(g, marks, kappa, pm, 0.07, 1.3, 0.01, ctx=gpu_ctx)
    for a in range(3):
        assert np.array_equal(got[a], want[a])
