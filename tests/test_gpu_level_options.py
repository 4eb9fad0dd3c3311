"""Options of a level that choose what its residual runs on: the stored operators at p = 1, the element
kernel of cd, the launch shapes of the tuner.

Tolerance of the residuals: 1e-12 of the largest value, as in test_gpu_parity.py."""
import numpy as np
import pytest

import hpb
from oracle.oracle import Oracle
from test_gpu_parity import relerr

pytestmark = pytest.mark.gpu


def _vec(arrays):
    return np.concatenate([a.ravel() for a in arrays])


@pytest.mark.parametrize("n", [7, 83, 84])
def test_stored_operators_are_applied_at_p1(n):
    """n = 7 and 84 lie on the two sides of the size that divides the two forms of a p = 1 stage, n = 83
    between the sizes of FP64 and FP32. The stored operators sum an element's products in another
    order than the matrix-free kernels: the residuals agree to rounding and are not the same bit by
    bit, in either precision."""
    pr = hpb.cd_sinsin(n=n, p=1, kcond=1e-2, src=0.7)
    a, b, o = pr.gpu(), pr.gpu(), Oracle(pr)
    assert a.setup_preconditioner() == 0 and b.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    b.element_matrices(True)
    ns = pr.phys.nstage
    for prec, tol in ((0, 1e-12), (1, 1e-5)):
        a.rsdl(ns, prec)
        b.rsdl(ns, prec)
        o.rsdl(ns)
        assert relerr(b.residual(), o.residual()) < tol and relerr(a.residual(), o.residual()) < tol
        assert not np.array_equal(_vec(a.residual()), _vec(b.residual()))
    a.iterate(3)
    b.iterate(3)
    assert relerr(b.state(), a.state()) < 1e-11 and not np.array_equal(_vec(a.state()), _vec(b.state()))
    b.element_matrices(False)
    b.upload(pr.ugv, pr.ugs, pr.ugi)
    b.iterate(3)
    assert np.array_equal(_vec(a.state()), _vec(b.state()))
    a.close()
    b.close()


@pytest.mark.parametrize("p", [1, 2, 4])
def test_cd_returns_from_the_scalar_kernel(p):
    pr = hpb.cd_sinsin(n=7, p=p, kcond=1e-2, src=0.7)
    g, o = pr.gpu(), Oracle(pr)
    assert g.setup_preconditioner() == 0 and o.setup_preconditioner() == 0
    res = []
    for kind in (None, "scalar", "tensor"):
        if kind:
            g.element_kernel(kind)
        g.rsdl(pr.phys.nstage)
        o.rsdl(pr.phys.nstage)
        res.append(_vec(g.residual()))
        assert relerr(g.residual(), o.residual()) < 1e-12, kind
    assert np.array_equal(res[0], res[2])
    g.close()


@pytest.mark.parametrize("kind,p,tuned", [("ins", 1, False), ("ins", 4, False), ("cd", 2, False),
                                          ("scalar", 3, True), ("cylinder", 2, True)])
def test_tuner_keeps_shapes_that_no_kernel_reads(kind, p, tuned):
    """The CTAs an SM of the scalar kernel are tuned where it runs (asked for, or curved triangles),
    and stay at the default elsewhere, however the timings fall."""
    if kind == "cylinder":
        pr = hpb.channel_cylinder_ins(scale=8.0, p=p)
    else:
        pr = hpb.cd_sinsin(n=9, p=p, kcond=1e-2) if kind == "cd" else hpb.kovasznay_ins(n=9, p=p)
    g = pr.gpu()
    if kind == "scalar":
        g.element_kernel("scalar")
    assert g.setup_preconditioner() == 0
    default = {prec: t["elem_cap"] for prec, t in g.tuning().items()}
    for _ in range(4):
        t = g.autotune(reps=1)
        for prec in ("fp64", "fp32"):
            assert t[prec]["elem_ms"] > 0 and t[prec]["minv_ms"] > 0
            if tuned:
                assert t[prec]["elem_cap"] in (4, 8, 16)
            else:
                assert t[prec]["elem_cap"] == default[prec]
    g.close()
