"""Workloads of this library for timing: what a user's program has it do, through its public entry points.

Kinds (a case is a dict of plain values; ``kind`` says how to read it):

* ``run``      one solver stepped by ``step(n)`` or ``step_graph(n)``, then its macro fields (and statistics) read
               where they lie.  method legacy|home|hybrid, storage f32|f16|bf16|f64, a periodic box or a duct.
* ``dropin``   the same through the ``LBM3D_*`` classes with their defaults (the reference's bounce table,
               ``step`` synchronous), as a program moved over from the reference calls them.
* ``sweep``    many uneven Hybrid(B0) ducts advanced together by ``Batch``, statistics of every instance read.
* ``adjoint``  the drag of a duct and its gradient, through the torch function.
* ``vtk``      the text of one VTK field, formatted into device memory.
* ``setup``    a new geometry for a solver in hand: voxelize, solid mask, band, initial fields.

The sizes are those of the benchmark, the tests, the command-line tools' defaults and of ragged grids between
them.
"""
import ctypes
import math

import numpy as np
import torch

from myfluidsimulation_b200 import geometry, lib
from myfluidsimulation_b200 import workloads as W
from myfluidsimulation_b200._lib import VTK_SCALAR, VTK_SPEED, VTK_VECTOR, check
from myfluidsimulation_b200.adjoint import DuctProblem, drag_objective
from myfluidsimulation_b200.solvers import (BC_DUCT, BC_PERIODIC, METHOD_HOME, METHOD_HYBRID, METHOD_LEGACY,
                                            STORE_BF16, STORE_F16, STORE_F32, STORE_F64, Batch, Domain, LBM3D_Home,
                                            LBM3D_Hybrid, LBM3D_Legacy, Solver)

METHODS = {"legacy": METHOD_LEGACY, "home": METHOD_HOME, "hybrid": METHOD_HYBRID}
STORES = {"f32": STORE_F32, "f16": STORE_F16, "bf16": STORE_BF16, "f64": STORE_F64}
BYTES = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}
CLASSES = {"legacy": LBM3D_Legacy, "home": LBM3D_Home, "hybrid": LBM3D_Hybrid}
VTK_KINDS = {"scalar": VTK_SCALAR, "speed": VTK_SPEED, "vector": VTK_VECTOR}
U_IN = 0.05


def _run(name, method, storage, flow, nx, ny, nz, steps, graph=False, stats=False, b0=0, tau=0.56):
    return {"name": name, "kind": "run", "method": method, "storage": storage, "flow": flow, "nx": nx, "ny": ny,
            "nz": nz, "steps": steps, "graph": graph, "stats": stats, "b0": b0, "tau": tau}


def listed():
    return [
        # the smallest call: an interactive loop that steps once and looks at the fields
        _run("tgv32_legacy_step1", "legacy", "f32", "tgv", 32, 32, 32, 1, tau=0.6),
        # the accuracy test's grid, replayed from a graph by a program that steps often and reads seldom
        _run("tgv64_home_graph20", "home", "f32", "tgv", 64, 64, 64, 20, graph=True, tau=0.6),
        # the reference's own class at its default domain, with an obstacle
        {"name": "dropin_legacy_default", "kind": "dropin", "method": "legacy", "solid": True, "nx": 128, "ny": 128,
         "nz": 96, "steps": 10, "tau": 0.6},
        # the benchmark's duct (periodic in x, driven by a force), 50 steps between statistics
        _run("duct_legacy", "legacy", "f32", "channel", 256, 128, 128, 50, stats=True),
        # the same duct with inlet and outlet, moment form
        _run("duct_home_inlet", "home", "f32", "duct", 256, 128, 128, 50, stats=True),
        # a ragged duct in 16-bit storage with a near-wall band
        _run("ragged_hybrid_f16", "hybrid", "f16", "duct", 201, 93, 77, 20, stats=True, b0=3, tau=0.55),
        # the largest: a 512^3 vortex in FP32
        _run("tgv512_legacy", "legacy", "f32", "tgv", 512, 512, 512, 10, tau=0.51),
        # the moment form in 16 bits on a large box
        _run("tgv256_home_bf16", "home", "bf16", "tgv", 256, 256, 256, 10, tau=0.51),
        # the B0 sweep: uneven ducts side by side
        {"name": "sweep_hybrid12", "kind": "sweep", "count": 12, "grids": 1, "steps": 50, "storage": "f32"},
        # the gradient of the drag: forward, recomputation and reverse pass
        {"name": "adjoint_128x64x64", "kind": "adjoint", "nx": 128, "ny": 64, "nz": 64, "steps": 100, "window": 20,
         "every": 25, "tau": 0.6},
        # the velocity file of a snapshot of the benchmark's duct
        {"name": "vtk_vector_duct", "kind": "vtk", "field": "vector", "nx": 256, "ny": 128, "nz": 128},
        # a new obstacle for the benchmark's duct (icosphere of 5,120 triangles, twice refined coverage)
        {"name": "setup_duct_refine2", "kind": "setup", "nx": 256, "ny": 128, "nz": 128, "levels": 4, "refine": 2,
         "b0": 2},
    ]


def draw(rng):
    """One more case of the same ranges."""
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def dims(lo, hi, cells):
        while True:
            d = [logint(lo, hi) for _ in range(3)]
            if rng.random() < 0.4:
                d[0] = max(16, d[0] // 16 * 16)
            if d[0] * d[1] * d[2] <= cells:
                return dict(zip(("nx", "ny", "nz"), d))

    p = rng.random()
    if p < 0.58:
        method = rng.choice(["legacy", "home", "hybrid"])
        storage = rng.choice(["f32", "f32", "f16", "bf16", "f64"])
        flow = rng.choice(["tgv", "channel", "duct"])
        d = dims(16, 448, 1 << 25)
        n = d["nx"] * d["ny"] * d["nz"]
        steps = min(logint(1, 60), max(1, int(4e8 // n)))
        return {"kind": "run", "method": method, "storage": storage, "flow": flow, **d, "steps": steps,
                "graph": rng.random() < 0.3, "stats": rng.random() < 0.5,
                "b0": rng.choice([0, 1, 2, 3, 4, 6]) if method == "hybrid" else 0,
                "tau": round(rng.uniform(0.53, 0.8), 3)}
    if p < 0.68:
        return {"kind": "dropin", "method": rng.choice(["legacy", "home", "hybrid"]), "solid": rng.random() < 0.5,
                **dims(16, 256, 1 << 22), "steps": rng.choice([1, 2, 5, 10, 20]), "tau": round(rng.uniform(0.53, 0.8), 3)}
    if p < 0.76:
        return {"kind": "sweep", "count": rng.randint(2, 12), "grids": rng.randint(2, 1 << 20),
                "steps": rng.randint(2, 40), "storage": rng.choice(["f32", "f32", "f16", "bf16"])}
    if p < 0.84:
        steps = rng.randint(8, 100)
        return {"kind": "adjoint", **dims(16, 128, 1 << 19), "steps": steps, "window": rng.randint(1, max(1, steps // 4)),
                "every": rng.choice([5, 10, 25]), "tau": round(rng.uniform(0.55, 0.8), 3)}
    if p < 0.92:
        return {"kind": "vtk", "field": rng.choice(["scalar", "speed", "vector"]), **dims(16, 256, 1 << 22)}
    return {"kind": "setup", **dims(24, 256, 1 << 22), "levels": rng.randint(2, 4), "refine": rng.choice([1, 1, 2, 3]),
            "b0": rng.choice([1, 2, 4, 6])}


# ---- inputs ------------------------------------------------------------------

def _sphere(nx, ny, nz, radius=None):
    """Solid cells (nz, ny, nx) of a sphere in the front quarter of the grid."""
    r = radius if radius is not None else 0.125 * min(nx, ny, nz)
    z, y, x = np.meshgrid(np.arange(nz) + 0.5, np.arange(ny) + 0.5, np.arange(nx) + 0.5, indexing="ij", sparse=True)
    return ((x - nx / 4) ** 2 + (y - ny / 2) ** 2 + (z - nz / 2) ** 2 <= r * r).astype(np.uint8)


def _fields(nx, ny, nz, flow, seed, mask=None, u_in=U_IN):
    """rho, u, v, w (float32, on the GPU): a vortex of amplitude 0.05, or a duct's stream, with shear waves of
    random phase and strength and a little noise on top."""
    g = torch.Generator().manual_seed(1000003 * int(seed) + 17)
    ph = torch.rand(8, generator=g, dtype=torch.float64).tolist()
    am = (0.002 + 0.004 * torch.rand(4, generator=g, dtype=torch.float64)).tolist()
    dev = "cuda"
    ax = [2 * math.pi * (torch.arange(n, device=dev, dtype=torch.float64) + 0.5) / n for n in (nx, ny, nz)]
    X, Y, Z = ax[0].view(1, 1, -1), ax[1].view(1, -1, 1), ax[2].view(-1, 1, 1)
    if flow == "tgv":
        u = 0.05 * torch.sin(X) * torch.cos(Y) * torch.cos(Z)
        v = -0.05 * torch.cos(X) * torch.sin(Y) * torch.cos(Z)
        rho = 1 + 3 * 0.05 ** 2 / 16 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2)
    else:
        u = torch.full((nz, ny, nx), u_in if flow == "duct" else 0.02, device=dev, dtype=torch.float64)
        v = torch.zeros((nz, ny, nx), device=dev, dtype=torch.float64)
        rho = 1 + 0 * v
    tau = 2 * math.pi
    u = u + am[0] * torch.cos(Y + tau * ph[0]) * torch.cos(Z + tau * ph[1])
    v = v + am[1] * torch.cos(Z + tau * ph[2]) * torch.cos(X + tau * ph[3])
    w = am[2] * torch.cos(X + tau * ph[4]) * torch.cos(Y + tau * ph[5]) + 0 * rho
    rho = rho + 0.1 * am[3] * torch.cos(X + Y + tau * ph[6]) * torch.cos(Z + tau * ph[7])
    out = []
    gd = torch.Generator(device=dev).manual_seed(int(seed) + 5)
    for k, a in enumerate((rho, u, v, w)):
        a = a.to(torch.float32).contiguous()
        a += (1e-5 if k == 0 else 1e-4) * torch.randn(a.shape, generator=gd, device=dev, dtype=torch.float32)
        if mask is not None:
            a[torch.from_numpy(mask != 0).to(dev)] = 1.0 if k == 0 else 0.0
        out.append(a)
    return out


def _case_mask(case):
    if case["kind"] == "run" and case["flow"] == "tgv" or case["kind"] == "dropin" and not case["solid"]:
        return None
    d = (case["nx"], case["ny"], case["nz"])
    return _sphere(*d) if case["kind"] == "dropin" else W.duct_mask(*d, _sphere(*d))


def _force(case):
    if case["kind"] == "run" and case["flow"] == "duct":
        return (0.0, 0.0, 0.0)
    return (1e-5, 0.0, 0.0)


class _Addr:
    def __init__(self, ptr, shape, owner):
        self.owner = owner               # the fields live as long as the solver
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


class _Views:
    """Tensors over a solver's macro fields, one for each address it hands out.  A tensor keeps the solver alive."""

    def __init__(self, solver, shape):
        self.solver, self.shape, self.known = solver, shape, {}

    def __call__(self, ptrs):
        out = []
        for p in ptrs:
            t = self.known.get(p)
            if t is None:
                t = self.known[p] = torch.as_tensor(_Addr(p, self.shape, self.solver), device="cuda")
            out.append(t)
        return out


def _sweep_grids(case):
    """nx, ny, nz of each instance: the batched study's ranges."""
    r = np.random.default_rng(case["grids"])
    return [(int(r.choice(np.arange(64, 193, 16))), int(r.choice(np.arange(32, 97, 16))),
             int(r.choice(np.arange(32, 97, 16)))) for _ in range(case["count"])]


def _sweep_params(case, seed):
    r = np.random.default_rng(int(seed))
    return [{"tau": float(r.uniform(0.52, 0.8)), "b0": int(r.choice([0, 1, 2, 3, 4, 6])), "seed": int(r.integers(1 << 30))}
            for _ in range(case["count"])]


def _adjoint_inputs(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator().manual_seed(int(seed))
    ui = 0.04 + 0.002 * torch.randn((nz, ny), generator=g)
    u0 = 1e-3 * torch.randn((3, nz, ny, nx), generator=g)
    u0[0] += 0.04
    return ui.to("cuda"), u0.to("cuda")


def _mesh(case, seed):
    """The obstacle's triangles: a bumped icosphere, placed by the voxelizer's scale and translation."""
    d = (case["nx"], case["ny"], case["nz"])
    r = np.random.default_rng(int(seed))
    radius = 0.22 * min(d) * r.uniform(0.8, 1.0)
    stretch, scale, tr = W.duct_sphere_stl_params(*d, radius, (d[0] / 4, d[1] / 2, d[2] / 2))
    t = W.icosphere(case["levels"])
    k = r.uniform(2, 5, 3)
    t = t * (1 + 0.1 * np.sin(t @ np.diag(k)).sum(-1, keepdims=True) / 3)
    mesh = geometry.mesh_from_triangles((t * stretch).astype(np.float32))
    return mesh, geometry.VoxelParams(*d, scale, tr, case["refine"], 0.5)


class _State:
    """What a user's program holds: the handle, its inputs, and views of its fields."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        solvers, views = [], []
        for (nx, ny, nz), p in zip(_sweep_grids(case), _sweep_params(case, seed)):
            mask = W.duct_mask(nx, ny, nz, _sphere(nx, ny, nz, 0.15 * min(ny, nz)))
            s = Solver(nx, ny, nz, p["tau"], method=METHOD_HYBRID, storage=STORES[case["storage"]], bc=BC_DUCT,
                       inlet_u=0.04)
            s.set_solid_mask(mask)
            s.build_band(p["b0"])
            s.reinit_from_macro(*_fields(nx, ny, nz, "duct", p["seed"], mask, 0.04))
            solvers.append(s)
            views.append(_Views(s, (nz, ny, nx)))
        torch.cuda.synchronize()
        b = Batch(solvers)
        b.enable_stats(True)
        return _State(case=case, solvers=solvers, batch=b, views=views)
    if kind == "adjoint":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        mask = W.duct_mask(nx, ny, nz, _sphere(nx, ny, nz, 0.15 * min(nx, ny, nz)))
        prob = DuctProblem(nx, ny, nz, case["tau"], mask, n_steps=case["steps"],
                           window=(case["steps"] - case["window"] + 1, case["steps"]), checkpoint_every=case["every"])
        ui, u0 = _adjoint_inputs(case, seed)
        return _State(case=case, problem=prob, ui=ui.requires_grad_(), u0=u0.requires_grad_())
    if kind == "vtk":
        d = (case["nx"], case["ny"], case["nz"])
        f = _fields(*d, "duct", seed, W.duct_mask(*d, _sphere(*d)))
        n, k = d[0] * d[1] * d[2], VTK_KINDS[case["field"]]
        cap = lib().lbm_vtk_text_bound(k, n)
        abc = (f[0], None, None) if case["field"] == "scalar" else tuple(f[1:])
        return _State(case=case, what=k, n=n, cap=cap, abc=abc, text=torch.zeros(cap, dtype=torch.uint8, device="cuda"))
    d = (case["nx"], case["ny"], case["nz"])
    if kind == "setup":
        mesh, vox = _mesh(case, seed)
        s = Solver(*d, 0.56, method=METHOD_HYBRID, bc=BC_DUCT, inlet_u=U_IN)
        return _State(case=case, solver=s, mesh=mesh, vox=vox, fields=_fields(*d, "duct", seed),
                      views=_Views(s, (d[2], d[1], d[0])))
    mask = _case_mask(case)
    if kind == "dropin":
        s = CLASSES[case["method"]]()
        s.init(Domain(*d, case["tau"], *_force(case)))
        if mask is not None:
            s.setSolidMask(mask)
        f = _fields(*d, "tgv", seed, mask)
        s.reinitEquilibriumFromMacro(*f)
        return _State(case=case, solver=s, views=_Views(s, (d[2], d[1], d[0])))
    s = Solver(*d, case["tau"], _force(case), method=METHODS[case["method"]], storage=STORES[case["storage"]],
               bc=BC_DUCT if case["flow"] == "duct" else BC_PERIODIC, inlet_u=U_IN if case["flow"] == "duct" else 0.0)
    if mask is not None:
        s.set_solid_mask(mask)
    if case["method"] == "hybrid" and mask is not None:
        s.build_band(case["b0"])
    f = _fields(*d, case["flow"], seed, mask)
    s.reinit_from_macro(*f)
    s.enable_stats(case["stats"])
    s.synchronize()          # the inputs are not kept
    return _State(case=case, solver=s, views=_Views(s, (d[2], d[1], d[0])))


# ---- one pass ----------------------------------------------------------------

def _row(stats):
    """One row of a run's log."""
    return np.array(list(stats.values()), np.float32)


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "run":
        s = state.solver
        s.step_graph(case["steps"]) if case["graph"] else s.step(case["steps"])
        out = dict(zip(("rho", "u", "v", "w"), state.views(s.macro_ptrs())))
        if case["stats"]:
            out["stats"] = _row(s.stats())
        return out
    if kind == "dropin":
        s = state.solver
        s.step(case["steps"])
        return dict(zip(("rho", "u", "v", "w"), state.views((s.d_rho(), s.d_u(), s.d_v(), s.d_w()))))
    if kind == "sweep":
        state.batch.step(case["steps"])
        out = {"stats": state.batch.stats().astype(np.float32)}
        for i, (s, v) in enumerate(zip(state.solvers, state.views)):
            out["%02d" % i] = v(s.macro_ptrs())
        return out
    if kind == "adjoint":
        J = drag_objective(state.ui, state.u0, state.problem, "f32")
        gi, gu = torch.autograd.grad(J, (state.ui, state.u0))
        return {"J": float(J.detach()), "gi": gi, "gu": gu}
    if kind == "vtk":
        ln = ctypes.c_int64()
        p = [None if t is None else ctypes.c_void_p(t.data_ptr()) for t in state.abc]
        check(lib().lbm_vtk_format(state.what, *p, state.n, ctypes.c_void_p(state.text.data_ptr()), state.cap,
                                   ctypes.byref(ln), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"length": ln.value, "text": state.text}     # zeros behind the text
    s = state.solver
    body = geometry.voxelize_mesh_to_mask(state.mesh, state.vox)
    mask = W.duct_mask(case["nx"], case["ny"], case["nz"], body)
    s.set_solid_mask(mask)
    cells = s.build_band(case["b0"])
    s.reinit_from_macro(*state.fields)
    return {"mask": mask, "cells": cells, "band": s.band(), "fields": state.views(s.macro_ptrs())}


def work(case):
    """Bytes and operations that one pass cannot do without: the state read once and written once, the outputs
    written once, and the arithmetic of every step (about 250 operations per cell and BGK step, 350 in moment
    form, twice and four times that for the adjoint's reverse step)."""
    kind = case["kind"]
    if kind == "sweep":
        n = sum(a * b * c for a, b, c in _sweep_grids(case))
        return {"bytes": n * (2 * 19 * BYTES[case["storage"]] + 16 + 1), "flops": 250.0 * n * case["steps"]}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind in ("run", "dropin"):
        k = 10 if case["method"] == "home" else 19
        b = BYTES[case.get("storage", "f32")]
        macros = 0 if case["method"] == "home" and b == 4 else 16
        return {"bytes": n * (2 * k * b + macros), "flops": (350.0 if k == 10 else 250.0) * n * case["steps"]}
    if kind == "adjoint":
        return {"bytes": n * (1 + 3 * 4 + 3 * 4), "flops": 1250.0 * n * case["steps"]}
    if kind == "vtk":
        return {"bytes": n * (4 + 9 if case["field"] == "scalar" else 12 + (9 if case["field"] == "speed" else 27)), "flops": 0}
    tri = 20 * 4 ** case["levels"]
    return {"bytes": n * (1 + 1 + 1 + 4 + 16 + 76 + 16) + 36 * tri, "flops": 0}


# ---- the same in 64 bits -----------------------------------------------------

CX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0)
CY = (0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 0, 0, 0, 0, 1, -1, 1, -1)
CZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1)
OPP = (0, 2, 1, 4, 3, 6, 5, 10, 9, 8, 7, 14, 13, 12, 11, 18, 17, 16, 15)
OPP_REF = (0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 14, 13, 16, 15, 18, 17)   # the reference's bounce table
WQ = (1 / 3,) + (1 / 18,) * 6 + (1 / 36,) * 12


def _feq(q, rho, u, v, w, uu):
    cu = CX[q] * u + CY[q] * v + CZ[q] * w
    return WQ[q] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu)


def _dot(f, c):
    out = 0
    for q in range(19):
        if c[q] > 0:
            out = out + f[q]
        elif c[q] < 0:
            out = out - f[q]
    return out


class _Box:
    """Solid cells, links and the duct's ends of one case, for the 64-bit steps."""

    def __init__(self, mask, duct, u_in, shape):
        self.duct, self.u_in = duct, u_in
        self.solid = None if mask is None else torch.from_numpy(mask.reshape(shape) != 0).to("cuda")
        self.body = None if mask is None else torch.from_numpy((mask.reshape(shape) != 0) & ((mask.reshape(shape) & 8) == 0)).to("cuda")

    def pulled(self, a, q):
        """Values of `a` at x - c_q (periodic)."""
        return torch.roll(a, (CZ[q], CY[q], CX[q]), (0, 1, 2))

    def stream(self, fs, q, rho, table=OPP):
        """The population that arrives along q, given the post-collision ones and the cells' own density."""
        out = self.pulled(fs[q], q)
        if self.solid is not None:
            out = torch.where(self.pulled(self.solid, q), fs[table[q]], out)
        if self.duct and CX[q] > 0:
            r = rho if not isinstance(rho, float) else torch.full_like(out, rho)
            out = out.clone()
            out[..., 0] = WQ[q] * r[..., 0] * (1 + 3 * self.u_in + 3 * self.u_in ** 2)
        elif self.duct and CX[q] < 0:
            out = out.clone()
            out[..., -1] = fs[q][..., -1]
        return out

    def drag(self, fs, table=OPP):
        """Momentum that the links into the body exchange in this step."""
        d = [0.0, 0.0, 0.0]
        if self.body is None:
            return d
        for q in range(1, 19):
            hit = self.pulled(self.body, q) & ~self.solid       # the population arriving along q comes from the body
            if self.duct and CX[q]:
                hit[..., 0 if CX[q] > 0 else -1] = False
            v = float(fs[table[q]][hit].sum())
            for k, c in enumerate((CX, CY, CZ)):
                d[k] += (c[table[q]] - c[q]) * v
        return d

    def sums(self, rho, u, v, w, drag):
        live = torch.ones_like(rho, dtype=torch.bool) if self.solid is None else ~self.solid
        s = lambda a: float(a[live].sum())  # noqa: E731
        ke = s(0.5 * (u * u + v * v + w * w))
        return np.array([s(rho), ke, *drag, s(rho * u), s(rho * v), s(rho * w), ke / rho.numel()])

    def rest(self, rho, u, v, w):
        if self.solid is None:
            return rho, u, v, w
        z = torch.zeros((), dtype=torch.float64, device="cuda")
        return (torch.where(self.solid, 1 + z, rho), *[torch.where(self.solid, z, a) for a in (u, v, w)])


def _exact_bgk(box, fields, tau, force, steps, stats):
    rho, u, v, w = [a.double() for a in fields]
    uu = u * u + v * v + w * w
    f = [_feq(q, rho, u, v, w, uu) for q in range(19)]
    for n in range(steps):
        rho = sum(f[1:], f[0])
        u, v, w = (_dot(f, c) / rho + g for c, g in ((CX, force[0]), (CY, force[1]), (CZ, force[2])))
        if n == steps - 1 and not stats:
            break
        uu = u * u + v * v + w * w
        fs = f if box.solid is None else list(f)
        for q in range(19):
            fs[q] = f[q] + (_feq(q, rho, u, v, w, uu) - f[q]) / tau
        if n == steps - 1:
            break
        del uu
        if box.solid is None and not box.duct:
            for q in range(1, 19):
                fs[q] = box.pulled(fs[q], q)
            f = fs
        else:
            f = [torch.where(box.solid, f[q], box.stream(fs, q, rho)) if box.solid is not None else box.stream(fs, q, rho)
                 for q in range(19)]
    row = box.sums(rho, u, v, w, box.drag(fs)) if stats else None
    return box.rest(rho, u, v, w), row


def _exact_home(box, fields, tau, force, steps, stats, table):
    rho, u, v, w = [a.double() for a in fields]
    S = [torch.zeros_like(rho) for _ in range(6)]      # xx, xy, xz, yy, yz, zz
    k = 1 - 1 / tau
    for n in range(steps):
        B = [rho * u * u + k * S[0], rho * u * v + k * S[1], rho * u * w + k * S[2], rho * v * v + k * S[3],
             rho * v * w + k * S[4], rho * w * w + k * S[5]]
        tr = B[0] + B[3] + B[5]
        fs = []
        for q in range(19):
            x, y, z = CX[q], CY[q], CZ[q]
            cc = x * x * B[0] + y * y * B[3] + z * z * B[5] + 2 * (x * y * B[1] + x * z * B[2] + y * z * B[4])
            fs.append(WQ[q] * (rho + 3 * rho * (x * u + y * v + z * w) + 4.5 * cc - 1.5 * tr))
        f = [box.stream(fs, q, rho, table) for q in range(19)]
        drag = box.drag(fs, table) if stats and n == steps - 1 else None
        del B, tr, fs
        rho = sum(f[1:], f[0])
        u, v, w = (_dot(f, c) / rho + g for c, g in ((CX, force[0]), (CY, force[1]), (CZ, force[2])))

        def second(a, b):
            return sum(a[q] * b[q] * f[q] for q in range(19) if a[q] * b[q])

        S = [second(CX, CX) - rho / 3 - rho * u * u, second(CX, CY) - rho * u * v, second(CX, CZ) - rho * u * w,
             second(CY, CY) - rho / 3 - rho * v * v, second(CY, CZ) - rho * v * w, second(CZ, CZ) - rho / 3 - rho * w * w]
        del f
        rho, u, v, w = box.rest(rho, u, v, w)
        if box.solid is not None:
            S = [torch.where(box.solid, torch.zeros_like(a), a) for a in S]
    return (rho, u, v, w), (box.sums(rho, u, v, w, drag) if stats else None)


def _exact_adjoint(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ui, u0 = [a.double().requires_grad_() for a in _adjoint_inputs(case, seed)]
    mask = W.duct_mask(nx, ny, nz, _sphere(nx, ny, nz, 0.15 * min(nx, ny, nz)))
    box = _Box(mask, True, 0.0, (nz, ny, nx))
    tau, steps, first = case["tau"], case["steps"], case["steps"] - case["window"]
    hits = []
    for q in range(19):
        hit = box.pulled(box.body, q) & ~box.solid
        if CX[q]:
            hit[..., 0 if CX[q] > 0 else -1] = False
        hits.append(hit.double())

    def start(u):
        uu = (u * u).sum(0)
        return torch.stack([_feq(q, torch.ones_like(uu), u[0], u[1], u[2], uu) for q in range(19)])

    def step(f, inlet, counted):
        rho = f.sum(0)
        u, v, w = (_dot(f, c) / rho for c in (CX, CY, CZ))
        uu = u * u + v * v + w * w
        fs = [f[q] + (_feq(q, rho, u, v, w, uu) - f[q]) / tau for q in range(19)]
        out, drag = [], f.new_zeros(())
        for q in range(19):
            o = torch.where(box.pulled(box.solid, q), fs[OPP[q]], box.pulled(fs[q], q))
            if CX[q] > 0:
                o = torch.cat([(WQ[q] * rho[..., 0] * (1 + 3 * inlet + 3 * inlet * inlet))[..., None], o[..., 1:]], -1)
            elif CX[q] < 0:
                o = torch.cat([o[..., :-1], fs[q][..., -1:]], -1)
            out.append(torch.where(box.solid, f[q], o))
            if counted and CX[q]:
                drag = drag + (CX[OPP[q]] - CX[q]) * (fs[OPP[q]] * hits[q]).sum()
        return torch.stack(out), drag

    with torch.no_grad():
        states, J = [start(u0)], 0.0
        for n in range(steps):
            nxt, d = step(states[-1], ui, n >= first)
            J += float(d) / case["window"]
            if n < steps - 1:
                states.append(nxt)
    lam, gi = torch.zeros_like(states[0]), torch.zeros_like(ui)
    for n in range(steps - 1, -1, -1):
        f = states.pop().requires_grad_()
        inlet = ui.detach().requires_grad_()
        nxt, d = step(f, inlet, n >= first)
        obj = (nxt * lam).sum() + (d / case["window"] if n >= first else 0.0)
        lam, g = torch.autograd.grad(obj, (f, inlet))
        gi += g
    (gu,) = torch.autograd.grad((start(u0) * lam).sum(), u0)
    return {"J": J, "gi": gi, "gu": gu}


def exact(case, seed):
    """What ``run`` gives for these inputs, in 64-bit torch; None where the outputs are whole numbers and text, and
    for solid cells under the reference's bounce table in population form, whose slots keep older values."""
    kind = case["kind"]
    if kind in ("vtk", "setup"):
        return None
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    names = ("rho", "u", "v", "w")
    if kind == "sweep":
        out, rows = {}, []
        for i, ((nx, ny, nz), p) in enumerate(zip(_sweep_grids(case), _sweep_params(case, seed))):
            mask = W.duct_mask(nx, ny, nz, _sphere(nx, ny, nz, 0.15 * min(ny, nz)))
            m, row = _exact_bgk(_Box(mask, True, 0.04, (nz, ny, nx)), _fields(nx, ny, nz, "duct", p["seed"], mask, 0.04),
                                p["tau"], (0.0, 0.0, 0.0), case["steps"], True)
            out["%02d" % i] = list(m)
            rows.append(row[:8])
        out["stats"] = np.array(rows)
        return out
    d = (case["nx"], case["ny"], case["nz"])
    mask = _case_mask(case)
    if kind == "dropin" and mask is not None and case["method"] != "home":
        return None
    flow = case["flow"] if kind == "run" else "tgv"
    box = _Box(mask, flow == "duct", U_IN, (d[2], d[1], d[0]))
    fields = _fields(*d, flow, seed, mask)
    stats = kind == "run" and case["stats"]
    if case["method"] == "home":
        m, row = _exact_home(box, fields, case["tau"], _force(case), case["steps"], stats,
                             OPP if kind == "run" else OPP_REF)
    else:
        m, row = _exact_bgk(box, fields, case["tau"], _force(case), case["steps"], stats)
    out = dict(zip(names, m))
    if stats:
        out["stats"] = row
    return out
