"""A mesh whose last vertex belongs to no triangle, at p = 1 (both forms of the stage) and above. Such a
vertex has an empty range of incidences that starts past the end of the array, from which no kernel may
read; its own preconditioner is infinite (1 / 0) and its value undefined, the others are the oracle's.

Tolerance: as for the updates of the p = 1 stage (test_gpu_line.py), 1e-11 after two updates."""
import numpy as np
import pytest

import hpb
from oracle.oracle import Oracle
from test_gpu_line import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", ["ins", "cd"])
@pytest.mark.parametrize("p,n", [(1, 2), (1, 4), (1, 77), (2, 4), (3, 5)])
def test_vertex_without_triangles(physics, p, n):
    m = hpb.square_mesh(n)
    pr = _problem(hpb.Mesh(np.concatenate([m.pnts, [[2.0, 2.0]]]), m.tri_pnt), p, physics)
    g, o = pr.gpu(), Oracle(pr)
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    g.iterate(2)
    for _ in range(2):
        o.update()
    a, b = g.state(), o.state()
    a, b = (np.concatenate([x[0][:-1].ravel(), x[1].ravel(), x[2].ravel()]) for x in (a, b))
    assert np.all(np.isfinite(a))
    assert np.max(np.abs(a - b)) < 1e-11 * np.max(np.abs(b))
    g.close()
