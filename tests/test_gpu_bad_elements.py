"""A preconditioner set-up that meets bad elements inside a cycle (block::cycle stops where
setup_preconditioner sets err, tri_mesh/blocks.cpp:1279): the call reports HP_ESTATE and stops ahead of
that level's updates, so the levels above keep the states they had then and nothing is prolongated."""
import numpy as np
import pytest

import hpb
from hpb import _lib as L
from hpb import multigrid as MG

pytestmark = pytest.mark.gpu

HP_ESTATE = -5


def _inverted(n):
    """square_mesh(n) with one interior vertex moved across its neighbours."""
    m = hpb.square_mesh(n)
    pts = m.pnts.copy()
    v = (n // 2) * (n + 1) + n // 2
    pts[v] += 2.5 / n
    bad = hpb.Mesh(pts, m.tri_pnt)
    assert bad.area2().min() < 0 < m.area2().min()
    return bad


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _vcycle(H, vw=1):
    return H.lib.hp_gpu_vcycle(H.handles(), len(H.levels), vw, 2, 2, 1)


@pytest.mark.parametrize("vw", [1, 2])
@pytest.mark.parametrize("p", [1, 3])
def test_vcycle_stops_ahead_of_a_bad_coarse_level(p, vw):
    n = 6
    fine = hpb.kovasznay_ins(n=n, p=p)
    if p > 1:
        H = MG.Hierarchy([fine, hpb.kovasznay_ins(p=1, mesh=_inverted(n))], ["fine", "p"])
    else:  # h-level: the weights of the good mesh, the coarse triangles of the bad one
        H = MG.Hierarchy([fine, hpb.kovasznay_ins(n=n // 2, p=1)], ["fine", "h"])
        t = hpb.kovasznay_ins(p=1, mesh=_inverted(n // 2)).gpu(stream=H._stream.cuda_stream)
        f2c, c2f = H._keep[:2], H._keep[2:]
        L.check(H.lib.hp_gpu_mg_attach_h(t.h, H.levels[0].h, *[L.ptr(a) for a in (*f2c, *c2f)], 1.0), "attach")
        H.levels[1].close()
        H.levels[1] = t
    alone = fine.gpu()
    assert alone.setup_preconditioner() == 0
    alone.iterate(2)  # what the fine level does before it restricts
    before = alone.state()
    assert _vcycle(H, vw) == HP_ESTATE
    assert _same(H.levels[0].state(), before)
    # the coarse level holds the restricted state, no update of it
    coarse = H.levels[1].state()[0]
    if p > 1:
        assert np.array_equal(coarse, before[0])
    assert np.all(np.isfinite(coarse))
    H.close()
    alone.close()


def test_vcycle_leaves_a_bad_finest_level_as_it_was():
    pr = hpb.kovasznay_ins(p=2, mesh=_inverted(6))
    H = MG.Hierarchy([pr], ["fine"])
    u = H.levels[0].state()
    assert _vcycle(H) == HP_ESTATE
    assert _same(H.levels[0].state(), u)
    H.close()


@pytest.mark.parametrize("graph", [False, True])
def test_solve_stops_ahead_of_a_bad_coarse_level(graph):
    fine = hpb.kovasznay_ins(n=6, p=3)
    H = MG.Hierarchy([fine, hpb.kovasznay_ins(p=1, mesh=_inverted(6))], ["fine", "p"])
    alone = fine.gpu()
    assert alone.setup_preconditioner() == 0
    alone.iterate(2)
    with pytest.raises(RuntimeError):
        H.solve(drop=1e-8, max_cycles=5, graph=graph)
    assert _same(H.levels[0].state(), alone.state())
    H.close()
    alone.close()
