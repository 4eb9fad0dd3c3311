"""The interior phase of minvrt divides by its pivots and by the triangle's preconditioner
(setup_preconditioner.cpp:343-372), each quotient rounded once.

On two separate triangles with essential values all around, the vertex and side modes are zero and the
interior mode of p = 3 is res / idiag / idiag / tprcn, three IEEE divisions: equal bit by bit."""
import ctypes

import numpy as np
import pytest
import torch

import hpb
from hpb import _lib as L
from test_gpu_line import _problem

pytestmark = pytest.mark.gpu


def test_interior_mode_is_divided_exactly():
    pnts = [[0.0, 0.0], [0.7, 0.1], [0.2, 0.9], [2.0, 0.0], [3.0, 0.2], [2.4, 0.7]]
    pr = _problem(hpb.Mesh(pnts, [[0, 1, 2], [3, 4, 5]]), 3, "cd")
    g = pr.gpu()
    assert g.setup_preconditioner() == 0
    ptrs = [ctypes.c_void_p() for _ in range(6)]
    L.check(g.lib.hp_gpu_device_ptrs(g.h, *[ctypes.byref(q) for q in ptrs]), "device_ptrs")

    class Interior:
        __cuda_array_interface__ = {"shape": (2,), "typestr": "<f8", "data": (ptrs[5].value, False), "version": 2}

    res = torch.as_tensor(Interior(), device="cuda")
    pivot, tp = pr.tab.idiag[0][1], g.prcn()[2][:, 0]
    for r in np.random.default_rng(1).normal(size=(40, 2)):
        g.rsdl(pr.phys.nstage)
        res.copy_(torch.from_numpy(r))
        torch.cuda.synchronize()
        g.minvrt()
        v, s, i = g.residual()
        assert not np.any(v) and not np.any(s)
        assert np.array_equal(i[:, 0, 0], r / pivot / pivot / tp)
    g.close()
