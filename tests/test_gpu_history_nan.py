"""The residual history of a diverged level: a value that is not a number shows as such and is not
lost in the maximum, at both forms of a p = 1 stage, at each form of the vertex phase above, wherever
the vertex lies in its warp and block; a vertex without triangles, whose value is undefined, does not
enter."""
import numpy as np
import pytest

import hpb
from test_gpu_line import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", ["ins", "cd"])
@pytest.mark.parametrize("kernel", ["tensor", "scalar"])
@pytest.mark.parametrize("p,n", [(1, 6), (1, 83), (2, 6), (3, 6), (3, 84), (6, 5)])
def test_nan_shows_in_the_history(physics, kernel, p, n):
    pr = _problem(hpb.square_mesh(n), p, physics)
    g = pr.gpu()
    if kernel == "scalar":
        g.element_kernel("scalar")
    assert g.setup_preconditioner() == 0
    assert np.all(np.isfinite(g.iterate(2)))
    for at in range(n // 2 * (n + 1) + 1, n // 2 * (n + 1) + 4):  # interior vertices
        v = pr.ugv.copy()
        v[at, 0] = np.nan
        g.upload(v, pr.ugs, pr.ugi)
        assert np.all(np.isnan(g.iterate(2)))
    g.close()


@pytest.mark.parametrize("p,n", [(1, 6), (1, 83), (2, 6), (3, 84)])
def test_vertex_without_triangles_does_not_enter(p, n):
    m = hpb.square_mesh(n)
    a = _problem(m, p).gpu()
    b = _problem(hpb.Mesh(np.concatenate([m.pnts, [[2.0, 2.0]]]), m.tri_pnt), p).gpu()
    b.upload(np.concatenate([a.prob.ugv, b.prob.ugv[-1:]]), a.prob.ugs, a.prob.ugi)
    for g in (a, b):
        assert g.setup_preconditioner() == 0
    ha, hb = a.iterate(2), b.iterate(2)
    assert np.all(np.isfinite(hb)) and np.allclose(ha, hb, rtol=1e-12, atol=0)
    a.close()
    b.close()
