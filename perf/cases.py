"""Performance cases: the work a user of this framework has it do, through its public entry
points (hpb.Problem / GPULevel / Hierarchy, hpb.tet, hpb.learned.MLP, the C-ABI they bind).

The framework's main path is the multistage smoother of the hp-FEM Navier-Stokes and
convection-diffusion solvers and the multigrid cycle around it, in two and three dimensions.
The cases are its residual evaluations, its smoothing sweeps, its cycles and the inference of
the learned preconditioner, from a coarse level of a few hundred triangles (launch latency) to
the half-million-triangle cavity."""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hp-multiphysics_b200"))

import hpb  # noqa: E402
from hpb import _lib as L  # noqa: E402
from hpb import learned as LR  # noqa: E402
from hpb import multigrid as MG  # noqa: E402
from hpb import tet as TT  # noqa: E402
from hpb.tetmesh import cube_tets  # noqa: E402

# Smoother cfl of the convection-diffusion runs, by p (the sweeps of the repository's benchmark)
CD_CFL = {8: 0.3, 7: 0.3, 6: 0.35, 5: 0.4, 4: 0.5, 3: 0.6, 2: 0.75, 1: 1.0}


def listed():
    return [
        # the benchmark's step: one FP64 residual of the 524,288-triangle lid-driven cavity at p = 6
        {"name": "rsdl_cavity_p6_n512", "kind": "rsdl", "flow": "cavity", "p": 6, "n": 512},
        # the Kovasznay flow at p = 4 on 64 x 64 squares: a small problem's residual, where launches count
        {"name": "rsdl_kovasznay_p4_n64", "kind": "rsdl", "flow": "kovasznay", "p": 4, "n": 64},
        # p = 3 on an unstructured mesh of ragged size: every local orientation, odd triangle count
        {"name": "rsdl_kovasznay_p3_delaunay", "kind": "rsdl", "flow": "kovasznay_delaunay", "p": 3, "n": 183},
        # convection-diffusion from stored element operators on 200k Delaunay triangles (bandwidth)
        {"name": "rsdl_cd_p4_stored", "kind": "rsdl", "flow": "cd_stored", "p": 4, "n": 317},
        # smoothing sweeps of a fine Navier-Stokes level
        {"name": "sweeps_cavity_p6_n256", "kind": "sweeps", "flow": "cavity", "p": 6, "n": 256, "sweeps": 2},
        # smoothing sweeps past the cylinder: graded mesh, curved (isoparametric) hole sides, p = 4
        {"name": "sweeps_cylinder_p4", "kind": "sweeps", "flow": "cylinder", "p": 4, "n": 50, "sweeps": 4},
        # the smallest calls: the sweeps a cycle makes on a coarse p = 1 level of 512 triangles
        {"name": "sweeps_kovasznay_p1_n16", "kind": "sweeps", "flow": "kovasznay", "p": 1, "n": 16, "sweeps": 4},
        # one W-cycle of the cavity hierarchy in FP64: p-levels 6, 3, 1 and three h-levels
        {"name": "wcycle_cavity_p6_n256", "kind": "cycles", "flow": "cavity", "p": 6, "n": 256, "h": 3, "vw": 2,
         "cycles": 1},
        # convection-diffusion V-cycles, matrix-free, p = 2
        {"name": "vcycles_cd_p2_n201", "kind": "cycles", "flow": "cd", "p": 2, "n": 201, "h": 3, "vw": 1, "cycles": 2},
        # a whole solve: FP32 V-cycles inside FP64 defect correction to convergence
        {"name": "solve_mixed_p6_n128", "kind": "mixed", "flow": "kovasznay", "p": 6, "n": 128, "h": 4, "vw": 1},
        # smoothing sweeps of the three-dimensional path, p = 3 on 196,608 tetrahedra
        {"name": "tet_sweeps_p3_n32", "kind": "tet", "p": 3, "n": 32, "sweeps": 6},
        # inference of the learned preconditioner correction on every triangle of the cavity
        {"name": "mlp_forward_524k", "kind": "mlp", "n": 524288},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rsdl", "rsdl", "rsdl", "rsdl", "sweeps", "sweeps", "sweeps", "cycles", "mixed", "tet", "mlp"])
    if kind == "rsdl":
        p = rng.randint(1, 8)
        flow = rng.choice(["cavity", "kovasznay", "kovasznay_delaunay", "cd", "cd_stored"])
        top = {"cavity": 450, "kovasznay": 450, "kovasznay_delaunay": 250, "cd": 450, "cd_stored": 250}[flow]
        return {"kind": kind, "flow": flow, "p": p, "n": _log_int(rng, 8, top * min(1.0, 6.0 / p) * 0.8)}
    if kind == "sweeps":
        p = rng.randint(1, 8)
        flow = rng.choice(["cavity", "kovasznay", "cylinder", "cd", "cd_stored"])
        n = rng.randint(35, 100) if flow == "cylinder" else _log_int(rng, 8, 220 * min(1.0, 6.0 / p))
        return {"kind": kind, "flow": flow, "p": p, "n": n, "sweeps": rng.randint(1, 6)}
    if kind == "cycles":
        flow = rng.choice(["cavity", "kovasznay", "cd"])
        p = rng.choice([2, 3, 4, 6])
        return {"kind": kind, "flow": flow, "p": p, "n": _log_int(rng, 24, 180), "h": rng.randint(1, 3),
                "vw": 1 if flow == "cd" else 2, "cycles": 1}
    if kind == "mixed":
        n = rng.randint(24, 64)
        return {"kind": kind, "flow": "kovasznay", "p": rng.choice([4, 6]), "n": n, "h": int(math.log2(n / 8)), "vw": 2}
    if kind == "tet":
        return {"kind": kind, "p": rng.randint(1, 3), "n": _log_int(rng, 4, 30), "sweeps": rng.randint(2, 6)}
    return {"kind": kind, "n": _log_int(rng, 500, 524288)}


# --- inputs -----------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _mesh(flow, n):
    if flow in ("kovasznay_delaunay", "cd_stored"):
        return hpb.delaunay_square(n, seed=20261205 + n)
    if flow == "cylinder":  # n: edge length at the hole in thousandths (the graded channel mesh scales with it)
        s = n / 20.0
        return hpb.channel_hole(hmin=0.02 * s, hmax=0.2 * s, grade=0.0085 * s)
    return hpb.square_mesh(n)


@functools.lru_cache(maxsize=None)
def _tets(n):
    return cube_tets(n)


def _problem(flow, n, p, seed, mesh=None):
    """The flow's problem with its initial state: the field projected on the basis plus 1e-3
    seeded noise on every coefficient, boundary values set."""
    mesh = _mesh(flow, n) if mesh is None else mesh
    if flow == "cavity":
        return hpb.lid_cavity_ins(n=n, p=p, re=400.0, mesh=mesh, seed=seed)
    if flow.startswith("kovasznay"):
        return hpb.kovasznay_ins(n=n, p=p, re=100.0, mesh=mesh, seed=seed)
    if flow == "cylinder":
        return hpb.channel_cylinder_ins(p=p, re=100.0, mesh=mesh, seed=seed)
    return hpb.cd_sinsin(n=n, p=p, mesh=mesh, seed=seed, cfl=CD_CFL[p])


class _DeviceArray:
    """A device buffer of a level as a torch tensor, without a copy; the tensor keeps the level open."""

    def __init__(self, address, shape, level):
        self.level = level
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (address, False), "version": 2}


def _views(level):
    """The level's state and residual on the device: ({"v", "s", "i"}, {"v", "s", "i"})."""
    ptrs = [ctypes.c_void_p() for _ in range(6)]
    L.check(level.lib.hp_gpu_device_ptrs(level.h, *[ctypes.byref(q) for q in ptrs]), "device_ptrs")
    pr = level.prob
    out = []
    for k in (0, 3):
        out.append({name: torch.as_tensor(_DeviceArray(ptrs[k + j].value, a.shape, level), device="cuda")
                    for j, (name, a) in enumerate((("v", pr.ugv), ("s", pr.ugs), ("i", pr.ugi))) if a.size})
    return out


def _mlp_inputs(n, seed):
    """Standardised element features [n][17] and the network of the learned correction."""
    rng = np.random.default_rng(seed)
    x = rng.normal(0.0, 1.0, (n, 17)).astype(np.float32) * np.linspace(0.5, 3.0, 17, dtype=np.float32)
    mean = rng.normal(0.0, 0.1, 17).astype(np.float32)
    std = rng.uniform(0.5, 2.0, 17).astype(np.float32)
    widths = (17, 64, 64, 64, 1)
    params = []
    for a, b in zip(widths[:-1], widths[1:]):
        params.append(rng.uniform(-1, 1, (b, a)).astype(np.float32) * np.float32(math.sqrt(6.0 / a)))
        params.append(rng.uniform(-0.1, 0.1, b).astype(np.float32))
    return x, mean, std, widths, params


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        x, mean, std, widths, params = _mlp_inputs(case["n"], seed)
        net = LR.MLP(widths)
        net.set_norm(mean, std)
        net.set_params(np.concatenate([a.ravel() for a in params]))
        return {"kind": kind, "net": net, "x": torch.from_numpy(x).cuda(), "n": case["n"]}
    if kind == "tet":
        n, p = case["n"], case["p"]
        pr = TT.TetProblem(_tets(n), p, mu=0.01, cfl=0.5).set_beltrami(re=100.0, seed=seed)
        masks, faces = pr.cube_boundary(re=100.0)
        g = TT.TetGPU(pr)
        g.set_dirichlet(masks)
        g.set_flux_faces(faces)
        if g.setup_preconditioner():
            raise RuntimeError("bad tetrahedra")
        g.jacobian_diagonal()
        return {"kind": kind, "level": g, "sweeps": case["sweeps"]}
    flow, n, p = case["flow"], case["n"], case["p"]
    if kind in ("cycles", "mixed"):
        stream = torch.cuda.Stream()
        levels = [(n, q, "p") for q in [p] + MG.p_sequence(p)] + [(n >> k, 1, "h") for k in range(1, case["h"] + 1)]
        h = MG.Hierarchy([_problem(flow, m, q, seed) for m, q, _ in levels], [k for _, _, k in levels],
                         stream=ctypes.c_void_p(stream.cuda_stream))
        h._stream = stream
        top = h.probs[0]
        return {"kind": kind, "h": h, "vw": case["vw"], "cycles": case.get("cycles", 0),
                "start": (top.ugv, top.ugs, top.ugi), "out": _views(h.levels[0])[0]}
    g = _problem(flow, n, p, seed).gpu()
    g.setup_preconditioner()
    if flow == "cd_stored":
        g.element_matrices(True)
    state, res = _views(g)
    return {"kind": kind, "level": g, "state": state, "res": res, "sweeps": case.get("sweeps", 0)}


# --- one pass ---------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "rsdl":  # the full residual, stream-ordered as a host solver enqueues it
        g = state["level"]
        L.check(g.lib.hp_gpu_enqueue_rsdl(g.h, g.prob.phys.nstage), "rsdl")
        return state["res"]
    if kind == "sweeps":  # multistage updates back to back, with their residual history
        hist = state["level"].iterate(state["sweeps"])
        return {"hist": hist, **state["state"]}
    if kind == "cycles":  # whole multigrid cycles with their preconditioner set-ups and norms
        state["h"].solve(drop=1e-30, max_cycles=state["cycles"], vw=state["vw"])
        return state["out"]
    if kind == "mixed":  # from the initial state to convergence
        state["h"].levels[0].upload(*state["start"])
        state["h"].solve(drop=1e-12, max_cycles=240, vw=state["vw"], mixed=True)
        # one vector: the converged flow is smooth, its high modes are small beside the rest
        return torch.cat([a.reshape(-1) for a in state["out"].values()])
    if kind == "tet":  # sweeps, then the state back to the host (the level's only way out)
        g = state["level"]
        g.iterate(state["sweeps"])
        return [a for a in g.state() if a.size]
    y = torch.empty((state["n"], 1), dtype=torch.float32, device="cuda")
    state["net"].forward(state["x"].data_ptr(), y.data_ptr(), state["n"],
                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return y


# --- what a pass cannot do without ------------------------------------------------------

def _entities(flow, n):
    if flow in ("kovasznay_delaunay", "cd_stored", "cylinder"):
        m = _mesh(flow, n)
        return m.npnt, m.nseg, m.ntri
    return (n + 1) ** 2, 3 * n * n + 2 * n, 2 * n * n


def _level_work(flow, n, p):
    """(coefficients, mesh bytes, flops of the imaginary part, flops of the real part) of a
    level's residual, in the sum-factorised form of the basis operators."""
    npnt, nseg, ntri = _entities(flow, n)
    cd = flow.startswith("cd")
    nv, nd = (1, 1) if cd else (3, 2)
    g, x, t = p + 1, p + 2, (p + 1) * (p + 2) // 2
    gg = g * g
    ndof = nv * (npnt + nseg * (p - 1) + ntri * (p - 1) * (p - 2) // 2)
    mesh = 36 * ntri + 16 * npnt
    if flow == "cd_stored":
        return ndof, mesh, ntri * 2 * t * t, ntri * 2 * t * t
    part = nv * (4 * x * gg + 4 * t * g)  # intgrtrs of one part
    im = nv * (2 * t * g + 2 * x * gg) + part + (5 if cd else 21) * gg
    re = nd * (2 * t * g + 4 * x * gg) + part + nv * gg * 6 * g + (20 if cd else 100) * gg
    return ndof, mesh, ntri * im, ntri * re


def _sweep_flops(flow, n, p):
    """One five-stage update: five imaginary parts, three real parts, five preconditioner solves."""
    ndof, mesh, im, re = _level_work(flow, n, p)
    npnt, nseg, ntri = _entities(flow, n)
    nv = 1 if flow.startswith("cd") else 3
    sm, inn = p - 1, (p - 1) * (p - 2) // 2
    minvrt = nv * (2 * (2 * nseg * sm + 3 * ntri * inn) + ntri * (2 * 3 * sm * (inn + 3 + 3 * (sm - 1) / 2.0) +
                                                                2 * (3 + 3 * sm) * inn + 5 * inn))
    return 5 * im + 3 * re + 5 * minvrt


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        n = case["n"]
        return {"bytes": n * 18 * 4 + 4 * 9473, "flops": 2.0 * n * (17 * 64 + 2 * 64 * 64 + 64)}
    if kind == "tet":
        n, p = case["n"], case["p"]
        ntet, npnt = 6 * n ** 3, (n + 1) ** 3
        nseg, ntri = 7 * n ** 3 + 9 * n * n + 3 * n, 12 * n ** 3 + 6 * n * n
        g, t = p + 1, (p + 1) * (p + 2) * (p + 3) // 6
        em, fm = p - 1, (p - 1) * (p - 2) // 2
        ndof = 4 * (npnt + nseg * em + ntri * fm + ntet * (t - 4 - 6 * em - 4 * fm))
        x = p + 3
        line = 2 * (t * g + x * x * g * g / 2 + x * g ** 3)  # one contraction, one direction after another
        im = 4 * line + 4 * 3 * line + 40 * g ** 3
        re = 3 * 3 * line + 4 * 3 * line + 4 * 6 * 2 * g ** 4 + 250 * g ** 3
        return {"bytes": 16 * ndof + 100 * ntet, "flops": float(case["sweeps"] * ntet * (5 * im + 3 * re))}
    flow, n, p = case["flow"], case["n"], case["p"]
    ndof, mesh, im, re = _level_work(flow, n, p)
    if kind == "rsdl":
        stored = 0
        if flow == "cd_stored":  # the operators are this path's input
            t = (p + 1) * (p + 2) // 2
            stored = _entities(flow, n)[2] * (2 * t * t + t) * 8
        return {"bytes": 16 * ndof + mesh + stored, "flops": im + re}
    if kind == "sweeps":
        return {"bytes": 16 * ndof + mesh, "flops": case["sweeps"] * _sweep_flops(flow, n, p)}
    # cycles: four sweeps per visit (two on the coarsest), each level visited vw times as often
    levels = [(n, q) for q in [p] + MG.p_sequence(p)] + [(n >> k, 1) for k in range(1, case["h"] + 1)]
    flops = 0.0
    for k, (m, q) in enumerate(levels):
        visits = case["vw"] ** min(k + 1, len(levels) - 1)
        flops += visits * (4 if k < len(levels) - 1 else 2 * case["vw"]) * _sweep_flops(flow, m, q)
    cycles = case["cycles"] if kind == "cycles" else (60 if case["vw"] == 2 else 150)  # a solve takes about that many
    return {"bytes": 16 * ndof + mesh, "flops": cycles * flops}


# --- results in 64 bits -----------------------------------------------------------------
# The residual of both physics written out densely: every triangle's modes evaluated at the
# tensor-product Gauss points of the collapsed coordinates, fluxes at the points, integrals
# against the test functions' derivatives.

def _gauss(n, al):
    """Gauss nodes and weights for the weight (1 - x)^al on [-1, 1] (Golub-Welsch)."""
    k = np.arange(n, dtype=np.float64)
    a = -al * al / ((2 * k + al) * (2 * k + al + 2)) if al else np.zeros(n)
    if al:
        a[0] = -al / (al + 2.0)
    k = k[1:]
    t = 2 * k + al
    b = 4 * k * (k + al) * k * (k + al) / (t * t * (t + 1) * (t - 1))
    lam, vec = np.linalg.eigh(np.diag(a) + np.diag(np.sqrt(b), 1) + np.diag(np.sqrt(b), -1))
    return lam, 2.0 ** (al + 1) / (al + 1) * vec[0] ** 2


def _monic(n, al, be, x):
    """Values and derivatives of the monic Jacobi(al, be) polynomials of degree 0 .. n - 1."""
    s = al + be
    v, d = [np.ones_like(x)], [np.zeros_like(x)]
    pm, dm, b = np.zeros_like(x), np.zeros_like(x), 0.0
    for k in range(n - 1):
        t = 2.0 * k + s
        a = (be - al) / (s + 2.0) if k == 0 else (be * be - al * al) / (t * (t + 2))
        if k == 1:
            b = 4.0 * (al + 1) * (be + 1) / ((s + 3.0) * (s + 2.0) ** 2)
        elif k > 1:
            b = 4.0 * k * (k + al) * (k + be) * (k + s) / (t * t * (t + 1) * (t - 1))
        v.append((x - a) * v[-1] - b * pm)
        d.append(v[-2] + (x - a) * d[-1] - b * dm)
        pm, dm = v[-2], d[-2]
    return v, d


@functools.lru_cache(maxsize=None)
def _basis(p):
    """Values and r, s derivatives of the modes at the points, weights, and the interpolation
    derivatives of point values: arrays over (mode, x point, eta point)."""
    g, sm = p + 1, p - 1
    x, wx = _gauss(g, 0)
    e, we = _gauss(g, 1)
    we = we / 2
    sx, dsx = _monic(max(sm, 1), 2.0, 2.0, x)
    se, dse = _monic(max(sm, 1), 2.0, 2.0, e)
    side_x = [((1 + x) * (1 - x) / 4 * q, -x / 2 * q + (1 + x) * (1 - x) / 4 * dq) for q, dq in zip(sx, dsx)][:sm]
    nrm = [1.0 / math.sqrt(np.sum(wx * f * f)) for f, _ in side_x]
    one, zero, half = np.ones(g), np.zeros(g), 0.5 * np.ones(g)
    fx = [(one, zero), ((1 - x) / 2, -half), ((1 + x) / 2, half)] + [(f * c, d * c) for (f, d), c in zip(side_x, nrm)]
    modes = [(0, (1 + e) / 2, half), (1, (1 - e) / 2, -half), (2, (1 - e) / 2, -half)]
    for m in range(2, sm + 2):
        modes.append((m + 1, ((1 - e) / 2) ** m, -m / 2 * ((1 - e) / 2) ** (m - 1)))
    for col, alt in ((2, 1), (1, -1)):
        for k in range(sm):
            sg = (alt ** k) * nrm[k]
            modes.append((col, sg * (1 - e) * (1 + e) / 4 * se[k], sg * (-e / 2 * se[k] + (1 - e) * (1 + e) / 4 * dse[k])))
    for m in range(2, sm + 1):
        v, d = _monic(sm + 1 - m, 2.0 * m + 1, 2.0, e)
        for q, dq in zip(v, d):
            f = ((1 - e) / 2) ** m * (1 + e) / 2 * q
            df = -m / 4 * ((1 - e) / 2) ** (m - 1) * (1 + e) * q + ((1 - e) / 2) ** m / 2 * (q + (1 + e) * dq)
            c = 1.0 / math.sqrt(np.sum(we * f * f))
            modes.append((m + 1, f * c, df * c))
    val = np.array([np.outer(fx[c][0], f) for c, f, _ in modes])
    dr = np.array([np.outer(fx[c][1], f * 2 / (1 - e)) for c, f, _ in modes])
    ds = np.array([np.outer(fx[c][0], df) for c, _, df in modes]) + (1 + x)[None, :, None] / 2 * dr

    def lagrange(z):
        w = np.array([np.prod(z[i] - np.delete(z, i)) for i in range(g)])
        m = np.array([[w[i] / (w[j] * (z[i] - z[j])) if i != j else 0.0 for j in range(g)] for i in range(g)])
        return m - np.diag(m.sum(1))

    dx = lagrange(x)[:, None, :, None] * np.eye(g)[None, :, None, :] * (2 / (1 - e))[None, :, None, None]
    de = np.eye(g)[:, None, :, None] * lagrange(e)[None, :, None, :] + (1 + x)[:, None, None, None] / 2 * dx
    q = g * g
    shape = lambda a: torch.from_numpy(np.ascontiguousarray(a.reshape(len(modes), q)))  # noqa: E731
    # the side functions at the x points: end 0, end 1, side modes
    ends = np.array([f for f, _ in fx[1:]])
    return (shape(val), shape(dr), shape(ds), torch.from_numpy(np.outer(wx, we).ravel()),
            torch.from_numpy(dx.reshape(q, q)), torch.from_numpy(de.reshape(q, q)), ends, wx)


def _exact_rsdl(pr):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m, p, nv = pr.mesh, pr.p, pr.NV
    cd = nv == 1
    sm = p - 1
    val, dr, ds, w, diff_r, diff_s, ends, wx = _basis(p)
    val, dr, ds, w, diff_r, diff_s = (a.to(dev) for a in (val, dr, ds, w, diff_r, diff_s))
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    pnts, tp, ts, tg = to(m.pnts), to(m.tri_pnt).long(), to(m.tri_seg).long(), to(m.tri_sgn)
    uv, us, ui = to(pr.ugv), to(pr.ugs), to(pr.ugi)
    rv, rs, ri = torch.zeros_like(uv), torch.zeros_like(us), torch.zeros_like(ui)
    flip = torch.where(torch.arange(max(sm, 0), device=dev) % 2 == 1, -1.0, 1.0).double()
    ph = pr.phys
    for a in range(0, m.ntri, 32768):
        t = slice(a, min(a + 32768, m.ntri))
        tri, seg = tp[t], ts[t]
        sg = torch.where(tg[t][:, :, None] < 0, flip, torch.ones_like(flip))  # (nt, 3, sm)
        u = torch.cat([uv[tri], (us[seg] * sg[..., None]).reshape(len(tri), -1, nv), ui[t]], 1)  # (nt, T, nv)
        x = pnts[tri]
        d0, d1 = (x[:, 2] - x[:, 1]) / 2, (x[:, 0] - x[:, 1]) / 2  # d x / dr, d x / ds
        jac = d0[:, 0] * d1[:, 1] - d0[:, 1] * d1[:, 0]
        # contravariant: r component of a flux (fx, fy), s component
        to_r = lambda fx, fy: d1[:, 1, None] * fx - d1[:, 0, None] * fy  # noqa: E731
        to_s = lambda fx, fy: -d0[:, 1, None] * fx + d0[:, 0, None] * fy  # noqa: E731
        f = torch.einsum("tmn,mq->ntq", u, val)
        fr, fs = torch.einsum("tmn,mq->ntq", u, dr), torch.einsum("tmn,mq->ntq", u, ds)
        gx = (d1[:, 1, None] * fr - d0[:, 1, None] * fs) / jac[:, None]  # physical derivatives
        gy = (-d1[:, 0, None] * fr + d0[:, 0, None] * fs) / jac[:, None]
        e1, e2, e3 = x[:, 0] - x[:, 1], x[:, 1] - x[:, 2], x[:, 2] - x[:, 0]
        leng = [torch.linalg.norm(q, dim=1) for q in (e1, e2, e3)]
        if cd:
            fluxes = [(ph.rhocv * ph.ax * f[0] - ph.kcond * gx[0], ph.rhocv * ph.ay * f[0] - ph.kcond * gy[0])]
        else:
            mf = (ph.rho * f[0], ph.rho * f[1])
            fluxes = [(f[0] * mf[0] + f[2] - ph.mu * 2 * gx[0], f[0] * mf[1] - ph.mu * (gy[0] + gx[1])),
                      (f[1] * mf[0] - ph.mu * (gy[0] + gx[1]), f[1] * mf[1] + f[2] - ph.mu * 2 * gy[1]), mf]
        pair = [(to_r(*q), to_s(*q)) for q in fluxes]
        strong = [q[0] @ diff_r.T + q[1] @ diff_s.T for q in pair]
        if cd:
            area2 = 4 * jac  # twice the triangle's area
            h = area2 / (0.25 * (p + 1) ** 2 * torch.stack(leng).max(0).values)
            lam = math.hypot(ph.ax, ph.ay) + 1.5 * (ph.kcond / ph.rhocv) / h
            tau = ph.adis * h / (jac * lam)
            s = tau[:, None] * (strong[0] - jac[:, None] * ph.src)
            pair = [(pair[0][0] - to_r(ph.ax, ph.ay) * s, pair[0][1] - to_s(ph.ax, ph.ay) * s)]
        else:
            h = 4 * jac / sum(leng) / (0.25 * (p + 1) ** 2)
            q2 = f[0] ** 2 + f[1] ** 2
            gam = 3 * q2 + (2 * ph.mu / ph.rho / h[:, None]) ** 2
            tau = ph.adis * (h / jac)[:, None] / torch.sqrt(gam)
            s0, s1, s2 = tau * strong[0], tau * strong[1], torch.sqrt(q2) * tau * strong[2]
            u0, u1 = f[0], f[1]
            supg = [(2 * u0 * s0 + s2, u1 * s0 + u0 * s1), (u1 * s0 + u0 * s1, 2 * u1 * s1 + s2), (s0, s1)]
            pair = [(q[0] - to_r(*b), q[1] - to_s(*b)) for q, b in zip(pair, supg)]
        out = torch.stack([-(torch.einsum("tq,mq->tm", q[0] * w, dr) + torch.einsum("tq,mq->tm", q[1] * w, ds))
                           for q in pair], 2)
        if cd and ph.src:
            out[:, :, 0] -= ph.src * jac[:, None] * (val * w).sum(1)
        rv.index_add_(0, tri.reshape(-1), out[:, :3].reshape(-1, nv))
        if sm:
            rs.index_add_(0, seg.reshape(-1), (out[:, 3:3 + 3 * sm].reshape(len(tri), 3, sm, nv) * sg[..., None])
                          .reshape(-1, sm, nv))
        ri[t] = out[:, 3 + 3 * sm:]
    if not cd:  # fluxes through the boundary sides that have one
        b = pr.bseg[(pr.bkind & (15 << 8)) == L.HP_BC_FLUX_INS_GENERIC]
        pb = pr.bpibc[:len(pr.bseg)][(pr.bkind & (15 << 8)) == L.HP_BC_FLUX_INS_GENERIC]
        v0, v1 = m.seg_pnt[b, 0], m.seg_pnt[b, 1]
        lin = np.concatenate([pr.ugv[v0][:, None], pr.ugv[v1][:, None], pr.ugs[b]], 1)
        u = np.einsum("bmn,mk->nbk", lin, ends)
        d = (m.pnts[v1] - m.pnts[v0]) / 2
        mass = ph.rho * (u[0] * d[:, 1, None] - u[1] * d[:, 0, None])
        flux = np.stack([mass * u[0] + pb * d[:, 1, None], mass * u[1] - pb * d[:, 0, None], mass], 2)
        part = to(np.einsum("bkn,mk,k->bmn", flux, ends, wx))
        rv.index_add_(0, to(v0).long(), part[:, 0])
        rv.index_add_(0, to(v1).long(), part[:, 1])
        if sm:
            rs.index_add_(0, to(b).long(), part[:, 2:])
    return {k: a for k, a in (("v", rv), ("s", rs), ("i", ri)) if a.numel()}


def exact(case, seed):
    """The residuals and the network's outputs. The smoothed states have none: they are iterates
    of the preconditioner, whose definition is the framework's own static inversion."""
    if case["kind"] == "mlp":
        x, mean, std, widths, params = _mlp_inputs(case["n"], seed)
        bf = lambda a: torch.from_numpy(a).bfloat16().double()  # noqa: E731  (the network's weights are BF16)
        y = (torch.from_numpy(x).double() - torch.from_numpy(mean).double()) / torch.from_numpy(std).double()
        for k in range(len(widths) - 1):
            y = y @ bf(params[2 * k]).T + bf(params[2 * k + 1])
            if k < len(widths) - 2:
                y = torch.relu(y)
        return y
    if case["kind"] == "rsdl":
        return _exact_rsdl(_problem(case["flow"], case["n"], case["p"], seed))
    return None
