"""res_r of the tetrahedra at a small viscosity without stabilisation (adis = 0): the real part then is
the viscous terms alone, 1e-9 of the convective ones, and keeps its own relative accuracy.

Tolerance: as at mu = 0.01 (test_gpu_tet.py), 1e-12 of the largest value: both sides sum the same
products of mu, in another order, and no term of another size enters."""
import pytest

from hpb.tet import TetGPU, TetProblem
from hpb.tetmesh import cube_tets
from oracle.oracle import OracleTet
from test_gpu_tet import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mu", [1e-6, 1e-9])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_viscous_residual_at_small_viscosity(p, mu):
    pr = TetProblem(cube_tets(3), p, mu=mu, adis=0.0).set_beltrami()
    g, o = TetGPU(pr), OracleTet(pr)
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    for stage in (pr.phys.nstage, 0, 2):
        g.rsdl(stage)
        o.rsdl(stage)
        assert relerr(g.residual(), o.residual()) < 1e-12, f"res stage {stage}"
        assert relerr(g.residual(1), o.residual_r()) < 1e-12, f"res_r stage {stage}"
    g.close()
