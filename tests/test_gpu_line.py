"""The ins line kernel (k_rsdl_ins_line: batches of 32 triangles, one lane each, persistent CTAs)
against the oracle at the sizes where it can go wrong: one partly filled batch, one full batch, a
full batch and a remainder, and more batches than resident CTAs (the loop over batches with its
one-ahead gather and two-ahead connectivity, at every slot of the connectivity ring).

Tolerance: both sides sum the same terms of each output in other orders; the longest chain is
about T + 3 G^2 = 290 FP64 operations at p = 8, 290 x 1.1e-16 = 3e-14 of the largest term, and
terms cancel by at most a factor of ~30 in the noisy states used, hence 1e-12 of the largest
residual."""
import ctypes

import numpy as np
import pytest

import hpb
from hpb import _lib as L
from oracle.oracle import Oracle
from test_gpu_parity import relerr, staircase_mesh

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _problem(mesh, p):
    field = L.Field(L.HP_FIELD_KOVASZNAY, (ctypes.c_double * 4)(100.0, 0, 0, 0))
    b = mesh.boundary_segments()
    return hpb.Problem(mesh, p, L.HP_PHYS_INS, rho=1.0, mu=0.01, field=field,
                       bc=[(b[::2], 0b011 | L.HP_BC_FLUX_INS_GENERIC),
                           (b[1::2], L.HP_BC_FLUX_INS_GENERIC)]).tobasis(noise=1e-3, seed=5)


# (mesh, p): n^2 triangles of staircase_mesh(n), 2 n^2 of square_mesh(n); the last column needs two
# to five passes of the batch loop on 148 SMs
CASES = ([("stair", 1, p) for p in (2, 6)] + [("square", 4, p) for p in range(2, 9)] +
         [("stair", 7, p) for p in range(2, 9)] +
         [("square", n, p) for p, n in ((2, 171), (3, 145), (4, 121), (5, 109), (6, 101), (7, 75), (8, 75))])


@pytest.mark.parametrize("kind,n,p", CASES)
def test_line_kernel_matches_oracle_at_batch_edges(kind, n, p):
    pr = _problem(staircase_mesh(n) if kind == "stair" else hpb.square_mesh(n), p)
    g, o = pr.gpu(), Oracle(pr)
    g.element_kernel("tensor")
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    # res_r mixes at stage 2 (0 < beta < 1), is left alone at stage 1 (beta = 0)
    for stage in ((pr.phys.nstage, 0, 1, 2) if pr.mesh.ntri < 1000 else (0, 2)):
        g.rsdl(stage)
        o.rsdl(stage)
        assert relerr(g.residual(), o.residual()) < TOL, stage
    g.close()
