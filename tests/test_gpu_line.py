"""The line kernel of ins and cd (k_rsdl_line: batches of 32 triangles, one lane each, persistent CTAs)
against the oracle at the sizes where it can go wrong: one partly filled batch, one full batch, a
full batch and a remainder, and more batches than resident CTAs (the loop over batches with its
one-ahead gather and two-ahead connectivity, at every slot of the connectivity ring); and the p = 1
stage (k_stage_p1 on small levels, k_vert_p1 on larger ones) around the size that divides them and
at a vertex of more than eight triangles.

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


def _problem(mesh, p, physics="ins"):
    b = mesh.boundary_segments()
    if physics == "cd":
        field = L.Field(L.HP_FIELD_SINSIN, (ctypes.c_double * 4)(1.0, 0, 0, 0))
        return hpb.Problem(mesh, p, L.HP_PHYS_CD, kcond=1e-2, ax=1.0, ay=0.5, src=0.3, cfl=0.3, field=field,
                           bc=[(b, 0b1)]).tobasis(noise=1e-3, seed=5)
    field = L.Field(L.HP_FIELD_KOVASZNAY, (ctypes.c_double * 4)(100.0, 0, 0, 0))
    return hpb.Problem(mesh, p, L.HP_PHYS_INS, rho=1.0, mu=0.01, field=field,
                       bc=[(b[::2], 0b011 | L.HP_BC_FLUX_INS_GENERIC),
                           (b[1::2], L.HP_BC_FLUX_INS_GENERIC)]).tobasis(noise=1e-3, seed=5)


# (mesh, p): n^2 triangles of staircase_mesh(n), 2 n^2 of square_mesh(n); the last column needs two
# to five passes of the batch loop on 148 SMs
CASES = ([("stair", 1, p) for p in (2, 6)] + [("square", 4, p) for p in range(1, 9)] +
         [("stair", 7, p) for p in range(1, 9)])
MANY = [("square", n, p) for p, n in ((1, 200), (2, 171), (3, 145), (4, 121), (5, 109), (6, 101), (7, 75), (8, 75))]
MANY_CD = [("square", n, p) for p, n in ((1, 215), (2, 200), (4, 150), (6, 120), (8, 80))]


@pytest.mark.parametrize("physics,kind,n,p", [("ins",) + c for c in CASES + MANY] +
                         [("cd",) + c for c in CASES + MANY_CD])
def test_line_kernel_matches_oracle_at_batch_edges(physics, kind, n, p):
    pr = _problem(staircase_mesh(n) if kind == "stair" else hpb.square_mesh(n), p, physics)
    g, o = pr.gpu(), Oracle(pr)
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    # res_r mixes at stage 2 (0 < beta < 1), is left alone at stage 1 (beta = 0)
    for stage in ((pr.phys.nstage, 0, 1, 2) if pr.mesh.ntri < 1000 else (0, 2)):
        g.rsdl(stage)
        o.rsdl(stage)
        assert relerr(g.residual(), o.residual()) < TOL, stage
    g.close()


@pytest.mark.parametrize("kind,n,p", [("stair", 1, 2), ("stair", 7, 3)] + [("square", 4, p) for p in range(2, 9)] +
                         [("square", n, p) for p, n in ((1, 16), (1, 83), (1, 84), (2, 216), (3, 141), (6, 100))])
def test_fp32_correction_update_matches_fp64_update(kind, n, p):
    """The FP32 line kernel in correction form (and k_base_points): one update of the FP32 smoother
    on the correction equation from d = 0 against one FP64 update from the same state.

    Tolerance: the correction is five stages of FP32 residuals, each a sum of at most 290 terms with
    6e-8 rounding (1.7e-5), cancellation of a factor of 10 between its terms: 1e-3 of the largest
    correction with the stages together."""
    pr = _problem(staircase_mesh(n) if kind == "stair" else hpb.square_mesh(n), p)
    g = pr.gpu()
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


def _fan(n):
    """n triangles around one vertex."""
    a = 2 * np.pi * np.arange(n) / n
    pts = np.concatenate([[[0.5, 0.5]], 0.5 + 0.5 * np.stack([np.cos(a), np.sin(a)], 1)])
    k = np.arange(n)
    return hpb.Mesh(pts, np.stack([0 * k, 1 + k, 1 + (k + 1) % n], 1).astype(np.int32))


@pytest.mark.parametrize("physics", ["ins", "cd"])
@pytest.mark.parametrize("nstage", [1, 2, 5])
@pytest.mark.parametrize("mesh", [("fan", 9), ("fan", 19), ("stair", 1), ("square", 75), ("square", 77)])
def test_p1_updates_match_oracle(mesh, nstage, physics):
    """Updates at p = 1 against the oracle: 5776 and 6084 vertices lie on the two sides of the size
    that divides the two forms on 148 SMs (5920). Tolerance as TOL, three updates long."""
    m = {"fan": _fan, "stair": staircase_mesh, "square": hpb.square_mesh}[mesh[0]](mesh[1])
    pr = _problem(m, 1, physics)
    pr.phys.nstage = nstage
    for k in range(nstage, 8):
        pr.phys.alpha[k] = pr.phys.beta[k] = 1.0
    g, o = pr.gpu(), Oracle(pr)
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    hist = g.iterate(3)
    for k in range(3):
        o.update()
        assert abs(hist[k] - o.maxres()[0]) <= 1e-9 * o.maxres()[0]
    assert relerr(g.state(), o.state()) < 1e-11
    g.rsdl(nstage)
    o.rsdl(nstage)
    assert relerr(g.residual(), o.residual()) < 1e-9  # (the residual has dropped below its terms)
    g.close()


@pytest.mark.parametrize("physics,p,n", [("ins", p, n) for p in (2, 3, 4, 6) for n in (83, 84)] +
                         [("cd", 3, 84), ("ins", 2, 3), ("ins", 5, 5), ("cd", 7, 4)])
def test_update_at_the_two_forms_of_the_vertex_phase(physics, p, n):
    """An update (minvrt's vertex phase with wide and narrow lane groups: 7056 and 7225 vertices lie
    on the two sides of the size that divides them on 148 SMs, 7104) against the oracle, tolerance
    as above for a third of the updates."""
    pr = _problem(hpb.square_mesh(n), p, physics)
    g, o = pr.gpu(), Oracle(pr)
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    hist = g.iterate(1)
    o.update()
    assert abs(hist[0] - o.maxres()[0]) <= 1e-9 * o.maxres()[0]
    assert relerr(g.state(), o.state()) < 1e-11
    g.close()
