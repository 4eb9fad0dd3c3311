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


@pytest.mark.parametrize("kind,n,p", [("stair", 1, 2), ("stair", 7, 3)] + [("square", 4, p) for p in range(2, 9)] +
                         [("square", n, p) for p, n in ((2, 216), (3, 141), (6, 100))])
def test_fp32_correction_update_matches_fp64_update(kind, n, p):
    """The FP32 line kernel in correction form (and k_base_points): one update of the FP32 smoother
    on the correction equation from d = 0 against one FP64 update from the same state.

    Tolerance: the correction is five stages of FP32 residuals, each a sum of at most 290 terms with
    6e-8 rounding (1.7e-5), cancellation of a factor of 10 between its terms: 1e-3 of the largest
    correction with the stages together."""
    pr = _problem(staircase_mesh(n) if kind == "stair" else hpb.square_mesh(n), p)
    g = pr.gpu()
    g.element_kernel("tensor")
    assert g.setup_preconditioner() == 0
    g.iterate(1)
    u64 = g.state()
    g.upload(pr.ugv, pr.ugs, pr.ugi)
    g.solve(mixed=True, drop=1e-30, max_updates=1, inner=1)
    u32 = g.state()
    u0 = (pr.ugv, pr.ugs, pr.ugi)
    d = np.concatenate([(a - b).ravel() for a, b in zip(u64, u0)])
    e = np.concatenate([(a - b).ravel() for a, b in zip(u32, u64)])
    assert np.max(np.abs(e)) < 1e-3 * np.max(np.abs(d))
    g.close()
