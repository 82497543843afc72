"""The work that users of warpcfd_gb300 have it do, as cases that can be timed.

Three kinds of user stand behind them: one who runs a case with ``IncompressibleSolver``
(steady SIMPLE or transient PISO), one who serves many cases with ``CaseBatch``, and one who
writes a loop of their own with the field operators, terms and equations of ``FVM``.  The
sizes are those of this repository's configurations (the 64^2 cavity, the 400x80 channel, the
247k-cell prism/hex cylinder, the 128^3 cavity, the serving mix of 1,024 to 65,536 cells) and
of its tests (jittered, tetrahedral and mixed meshes), with odd ones between them.

Every pass starts from the same state, so that all passes do the same work: a solver is put
back to a checkpoint (``snapshot`` / ``restore``) and then steps on from there.  The
checkpoint is the case's start with a perturbed velocity field, as a restart from another
run's fields gives it; lid or inlet speed, perturbation, viscosities and sources come from
the seed.
"""
import math

import numpy as np
import torch

from warpcfd_gb300.batch import CaseBatch
from warpcfd_gb300.FV import FVM
from warpcfd_gb300.FV.implicit_Solvers import IncompressibleSolver
from warpcfd_gb300.FV.terms import ConvectionTerm, DdtTerm, DiffusionTerm, Equation, GradTerm
from warpcfd_gb300.preprocess import (Mesh, create_2D_grid, create_3D_grid, create_cylinder_channel_grid,
                                      define_boundary_walls, define_cylinder_group)
from warpcfd_gb300.serve import (SERVE_ATOL, SERVE_CG_VARIANT, SERVE_P_REFINE, SERVE_RTOL, MeshCache, Request,
                                 build_solver, make_request_mix)

DEVICE = "cuda"


# ---------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest mesh of the serving mix, run as an interactive user does: 20 outer
        # iterations replayed from a CUDA graph, residuals read twice; latency and launches
        dict(name="cavity_32_run", kind="solver", mesh="2d", nx=32, ny=32, channel=False, iters=20, graph=True),
        # the 64^2 cavity, the reference's own example, stepped eagerly
        dict(name="cavity_64", kind="solver", mesh="2d", nx=64, ny=64, channel=False, iters=10, graph=False),
        # the 400x80 channel: an ordinary 2D case whose pressure solve runs to its cap
        dict(name="channel_400x80", kind="solver", mesh="2d", nx=400, ny=80, channel=True, iters=2, graph=False),
        # a ragged, jittered tetrahedral box (four faces per cell, unstructured numbering)
        dict(name="cavity_tetra_23x19x21", kind="solver", mesh="tetra", nx=23, ny=19, nz=21, jitter=0.1, iters=3,
             graph=False),
        # an odd 3D box of ordinary size
        dict(name="cavity3d_61x47x53", kind="solver", mesh="hex", nx=61, ny=47, nz=53, jitter=0.0, iters=3,
             graph=False),
        # the largest steady case: the 128^3 cavity
        dict(name="cavity3d_128", kind="solver", mesh="hex", nx=128, ny=128, nz=128, jitter=0.0, iters=2,
             graph=False),
        # one PISO time step around a cylinder: prisms and hexes, non-orthogonal correction, two
        # correctors, fp64-refined pressure solves
        dict(name="cylinder_piso_247k", kind="piso", scale=1.15, refine=3),
        # one round (10 outer iterations) of the server's largest bucket and of its smallest
        dict(name="serve_large_8", kind="serve", lo=32769, hi=65536, count=8),
        dict(name="serve_small_48", kind="serve", lo=1024, hi=4096, count=48),
        # loops of a user's own: the momentum predictor and a Poisson equation with a face-wise
        # coefficient, assembled from terms and solved; the field operators alone
        dict(name="momentum_loop_83x64x48", kind="momentum", nx=83, ny=64, nz=48),
        dict(name="poisson_loop_96x90x100", kind="poisson", nx=96, ny=90, nz=100),
        dict(name="field_operators_112x121x104", kind="fields", nx=112, ny=121, nz=104),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """A box of about exp(U[log lo, log hi]) cells with sides within a factor of two."""
    n = _log_int(rng, lo, hi)
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    s = n ** (1.0 / 3.0)
    nx, ny = max(4, round(s * a)), max(4, round(s * b))
    return dict(nx=nx, ny=ny, nz=max(4, round(n / (nx * ny))))


def draw(rng):
    kind = rng.choice(["solver2d", "solver2d", "solver3d", "solver3d", "tetra", "piso", "serve", "momentum",
                       "poisson", "fields"])
    if kind == "solver2d":
        channel = rng.random() < 0.5
        n = _log_int(rng, 1024, 120000)
        ny = max(12, round(math.sqrt(n / (4.0 if channel else 1.0)) * rng.uniform(0.8, 1.25)))
        return dict(kind="solver", mesh="2d", nx=max(12, round(n / ny)), ny=ny, channel=channel,
                    iters=10 if n < 8000 else 2, graph=rng.random() < 0.5)
    if kind == "solver3d":
        return dict(kind="solver", mesh="hex", jitter=rng.choice([0.0, 0.1]), iters=2, graph=False,
                    **_box(rng, 4000, 1500000))
    if kind == "tetra":
        return dict(kind="solver", mesh="tetra", jitter=rng.choice([0.0, 0.1]), iters=2, graph=False,
                    **_box(rng, 700, 60000))
    if kind == "piso":
        return dict(kind="piso", scale=round(rng.uniform(0.3, 1.0), 3), refine=rng.choice([0, 1, 2, 3]))
    if kind == "serve":
        lo, hi, most = rng.choice([(1024, 4096, 48), (4097, 8192, 40), (8193, 16384, 32), (16385, 32768, 16),
                                   (32769, 65536, 8)])
        return dict(kind="serve", lo=lo, hi=hi, count=rng.randint(1, most))
    return dict(kind=kind, **_box(rng, 8000, 1400000))


# ------------------------------------------------------------------------- meshes and models
_meshes = {}   # the last mesh of a program that runs several cases on it
_ladder = []   # the serving meshes, kept as the server keeps them


def _mesh(case):
    kind = case["kind"]
    key = tuple(sorted((k, v) for k, v in case.items() if k in ("mesh", "nx", "ny", "nz", "jitter", "channel", "scale")))
    if key in _meshes:
        return _meshes[key]
    _meshes.clear()
    if kind == "piso":
        g, info = create_cylinder_channel_grid(scale=case["scale"], jitter=0.1, seed=0, prisms=True)
        m = Mesh(g, device=DEVICE)
        define_boundary_walls(m)
        define_cylinder_group(m, info["cylinder"])
    else:
        if case.get("mesh") == "2d":
            g = create_2D_grid((0, 0, 0), case["nx"], case["ny"], 10.0 if case["channel"] else 1.0, 1.0, 0.1)
        else:
            g = create_3D_grid((0, 0, 0), case["nx"], case["ny"], case["nz"], 1.0, 1.0, 1.0,
                               jitter=case.get("jitter", 0.0), seed=1,
                               element_type="tetra" if case.get("mesh") == "tetra" else "hex")
        m = Mesh(g, device=DEVICE)
        define_boundary_walls(m)
    _meshes[key] = m
    return m


def _modes(rng, pts, n):
    """n smooth scalar fields of order one at the points (N, 3): four sine modes each."""
    out = torch.zeros((pts.shape[0], n), dtype=torch.float64, device=pts.device)
    for f in range(n):
        for _ in range(4):
            k = torch.tensor(rng.uniform(-9.0, 9.0, 3), dtype=torch.float64, device=pts.device)
            out[:, f] += rng.uniform(-0.5, 0.5) * torch.sin(pts @ k + rng.uniform(0.0, 6.28))
    return out


def _centroids(model):
    return torch.as_tensor(np.ascontiguousarray(model.struct_member_to_array("centroid", "cells")),
                           dtype=torch.float64, device=DEVICE)


def _cavity_bc(b, lid):
    for w in ("-X", "+X", "-Y", "-Z", "+Z"):
        b.no_slip_wall(w)
    b.velocity_BC("+Y", u=lid, v=0.0, w=0.0)


def _solver_state(case, seed):
    rng = np.random.default_rng([seed, 1])
    speed = float(rng.uniform(0.8, 1.2))
    mesh = _mesh(case)
    model = FVM(mesh)
    b = model.boundary
    if case["kind"] == "piso":
        ids = mesh.groups["-X"].ids
        y = model.struct_member_to_array("centroid", "faces")[ids, 1]
        b.velocity_BC("-X", u=4.0 * 1.5 * speed * y * (0.41 - y) / 0.41 ** 2, v=0.0, w=0.0)
        b.pressure_BC("+X", p=0.0)
        for w in ("-Y", "+Y", "cylinder"):
            b.no_slip_wall(w)
        b.slip_wall("-Z")
        b.slip_wall("+Z")
        nu = 1e-3
    elif case["mesh"] == "2d" and case["channel"]:
        b.velocity_BC("-X", u=speed, v=0.0, w=0.0)
        b.pressure_BC("+X", p=0.0)
        for w in ("-Y", "+Y"):
            b.no_slip_wall(w)
        for w in ("-Z", "+Z"):
            b.slip_wall(w)
        nu = 1.0 / 200.0
    elif case["mesh"] == "2d":
        for w in ("-X", "+X", "-Y"):
            b.no_slip_wall(w)
        b.velocity_BC("+Y", u=speed, v=0.0, w=0.0)
        for w in ("-Z", "+Z"):
            b.slip_wall(w)
        nu = 0.01
    else:
        _cavity_bc(b, speed)
        nu = 1.0 / 400.0
    model.material.create_incompressible_newtonian_fluid(viscosity=nu, density=1.0)
    if case["kind"] == "solver" and not case.get("channel"):
        model.set_reference_pressure(0, 0.0)
    model.finalize()
    if case["kind"] == "piso":
        solver = IncompressibleSolver(model, None, None, correction=True, steady_state=False)
        solver.set_iterations(1, 2, 1)
        solver.set_time_stepping(1, 5e-4)
        solver.p_refine, solver.p_refine_rtol = case["refine"], 1e-3
    else:
        ur = 0.3 if case.get("channel") else 0.7
        solver = IncompressibleSolver(model, ur, 0.3, correction=case.get("jitter", 0.0) > 0.0)
        solver.set_iterations(case["iters"], 1, 1)
    solver.verbose = False
    ic = 0.1 * speed * _modes(rng, _centroids(model), 3)
    if case.get("mesh") == "2d" or case["kind"] == "piso":
        ic[:, 2] = 0.0
    model.set_initial_conditions(ic.float(), [0, 1, 2])
    solver.HbyA.copy_(ic.float().reshape(-1))
    solver.case_struct()
    return dict(case=case, model=model, solver=solver, start=solver.snapshot())


def _run_solver(st):
    case, model, solver = st["case"], st["model"], st["solver"]
    solver.restore(st["start"])
    if case.get("graph"):
        solver.run(steps_per_check=10, use_cuda_graph=True)
    else:
        for _ in range(case.get("iters", 1)):
            solver.step()
    return dict(cell_values=model.cell_values, cell_gradients=model.cell_gradients, face_values=model.face_values,
                mass_fluxes=model.mass_fluxes, HbyA=solver.HbyA, p=solver.p_corr_equation.x, rUA=solver.rUA)


# -------------------------------------------------------------------------------- serving
def _serve_state(case, seed):
    if not _ladder:
        _ladder.append(MeshCache(device=DEVICE))
    meshes = _ladder[0]
    # the sizes and kinds are the case's, Reynolds number and speed the seed's
    mix = make_request_mix(case["count"], seed=7, lo=case["lo"], hi=case["hi"])
    rng = np.random.default_rng([seed, 2])
    solvers, models = [], []
    for r in mix:
        cells = r.cells
        while np.prod(meshes.shape(r.kind, cells)) > case["hi"]:
            cells = int(cells * 0.95)
        req = Request(r.rid, r.kind, cells, float(rng.uniform(50.0, 1000.0)), float(rng.uniform(0.5, 2.0)), 0.0)
        model, solver = build_solver(req, meshes.get(r.kind, cells), atol=SERVE_ATOL, rtol=SERVE_RTOL,
                                     p_refine=SERVE_P_REFINE)
        model.set_initial_conditions((0.1 * req.speed * _modes(rng, _centroids(model), 2)).float(), [0, 1])
        solvers.append(solver)
        models.append(model)
    # the server's rule: the fewest CTAs per case that hold the bucket's largest case
    from warpcfd_gb300 import _lib
    rows = int(_lib.load().wcfd_batch_max_rows(4))
    cs = 1
    while cs * rows < case["hi"]:
        cs *= 2
    batch = CaseBatch(solvers, cluster_size=cs, cg_variant=SERVE_CG_VARIANT)
    tensors = [t for s in solvers for t in s.state_tensors()]
    return dict(case=case, batch=batch, models=models, tensors=tensors, start=[t.clone() for t in tensors],
                stream=torch.cuda.Stream())


def _run_serve(st):
    here = torch.cuda.current_stream()
    st["stream"].wait_stream(here)
    with torch.cuda.stream(st["stream"]):
        torch._foreach_copy_(st["tensors"], st["start"])
        st["batch"].steps(10)
    here.wait_stream(st["stream"])
    return [m.cell_values for m in st["models"]]


# ------------------------------------------------------------------- loops of a user's own
def _loop_inputs(case, seed):
    """Numbers of a loop case, from the seed alone, in 32 bits as the user holds them."""
    rng = np.random.default_rng([seed, 3])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x = (torch.arange(nx, dtype=torch.float64, device=DEVICE) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=DEVICE) + 0.5) / ny
    z = (torch.arange(nz, dtype=torch.float64, device=DEVICE) + 0.5) / nz
    Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
    pts = torch.stack([X.ravel(), Y.ravel(), Z.ravel()], dim=1)
    d = dict(lid=float(rng.uniform(0.8, 1.2)), values=_modes(rng, pts, 4).float())
    if case["kind"] == "poisson":
        g = torch.Generator(device=DEVICE)
        g.manual_seed(int(rng.integers(1 << 40)))
        K = 3 * nx * ny * nz + nx * ny + ny * nz + nx * nz
        d["kappa"] = 0.5 + torch.rand(K, generator=g, device=DEVICE, dtype=torch.float32)
        d["source"] = (d["values"][:, 0] + 0.1 * torch.randn(nx * ny * nz, generator=g, device=DEVICE)) / (nx * ny * nz)
    return d


MOMENTUM = dict(nu=1.0 / 400.0, rho=1.2, dt=0.05, relax=0.7)
POISSON_TOL = 1e-9


def _loop_state(case, seed):
    mesh = _mesh(case)
    d = _loop_inputs(case, seed)
    model = FVM(mesh)
    if case["kind"] == "poisson":
        b = model.boundary
        for w in ("-X", "-Y", "+Y", "-Z", "+Z"):
            b.slip_wall(w)
        b.pressure_BC("+X", p=0.0)
    else:
        _cavity_bc(model.boundary, d["lid"])
    model.finalize()
    model.set_initial_conditions(d["values"])
    st = dict(case=case, model=model, **d)
    if case["kind"] == "poisson":
        st["diffusion"], st["eq"] = DiffusionTerm(model, "p"), Equation(model, "p", solver="cg")
        st["eq"].tol = POISSON_TOL
    elif case["kind"] == "momentum":
        uvw = ["u", "v", "w"]
        st.update(convection=ConvectionTerm(model, uvw, "upwind"), diffusion=DiffusionTerm(model, uvw),
                  ddt=DdtTerm(model, uvw), grad=GradTerm(model, "p"), eq=Equation(model, uvw))
        st["eq"].tol = 1e-8
        st["x0"] = d["values"][:, :3].contiguous().reshape(-1)
    return st


def _run_fields(st):
    m = st["model"]
    m.set_boundary_conditions()
    m.face_interpolation()
    m.calculate_mass_flux()
    m.calculate_gradients()
    return dict(face_values=m.face_values, mass_fluxes=m.mass_fluxes, cell_gradients=m.cell_gradients, div=m.divFlux())


def _run_momentum(st):
    m, eq, c = st["model"], st["eq"], MOMENTUM
    m.set_boundary_conditions()
    m.face_interpolation()
    m.calculate_mass_flux()
    m.calculate_gradients()
    st["convection"](m)
    st["diffusion"](m, viscosity=c["nu"])
    st["ddt"](m, dt=c["dt"])
    st["grad"](m)
    eq.form_system([st["convection"], -st["diffusion"], st["ddt"]], -1.0 / c["rho"] * st["grad"])
    eq.relax(c["relax"])
    eq.x.copy_(st["x0"])
    eq.solve_Axb()
    return dict(diag=eq.diag, rhs=eq.rhs, x=eq.x)


def _run_poisson(st):
    m, eq = st["model"], st["eq"]
    m.set_boundary_conditions()
    st["diffusion"](m, viscosity=st["kappa"])
    eq.form_system(st["diffusion"])
    eq.add_RHS(st["source"])
    eq.x.zero_()
    eq.solve_Axb()
    return dict(diag=eq.diag, rhs=eq.rhs, x=eq.x)


# ----------------------------------------------------------------------------- prepare, run
def prepare(case, seed):
    if case["kind"] in ("solver", "piso"):
        return _solver_state(case, seed)
    if case["kind"] == "serve":
        return _serve_state(case, seed)
    return _loop_state(case, seed)


def run(state):
    return {"solver": _run_solver, "piso": _run_solver, "serve": _run_serve, "momentum": _run_momentum,
            "poisson": _run_poisson, "fields": _run_fields}[state["case"]["kind"]](state)


# -------------------------------------------------------------------------------- the work
def _counts(case):
    """(cells, faces, slots per cell, off-diagonals per row) of a case's mesh."""
    if case["kind"] == "piso":
        n = int(187000 * case["scale"] ** 2)
        return n, int(3.0 * n), 6, 4
    if case["kind"] == "serve":
        n = int(case["count"] * math.sqrt(case["lo"] * case["hi"]))
        return n, 4 * n, 6, 4
    nx, ny = case["nx"], case["ny"]
    if case.get("mesh") == "2d":
        n = nx * ny
        return n, 4 * n + nx + ny, 6, 4
    nz = case["nz"]
    n = nx * ny * nz
    if case.get("mesh") == "tetra":
        return 6 * n, 12 * n + 2 * (nx * ny + ny * nz + nx * nz), 4, 4
    return n, 3 * n + nx * ny + ny * nz + nx * nz, 6, 6


def work(case):
    C, K, F, W = _counts(case)
    geometry = 44 * K + (16 * F + 4) * C          # owner, neighbour, weights, normal, coefficient; slots, volume
    state = 64 * C + 36 * K                       # values and gradients of cells, values and gradients of faces, flux
    if case["kind"] == "fields":
        return dict(bytes=geometry + state + 4 * C, flops=70.0 * K + 24.0 * F * C)
    systems = (4 * W + 36) * C + (4 * W + 12) * C  # momentum and pressure, each written and read once
    if case["kind"] == "momentum":
        return dict(bytes=geometry + state + (4 * W + 36) * C, flops=70.0 * K + 60.0 * F * C + 8 * (6 * W + 60.0) * C)
    side = max(case.get("nx", 0), case.get("ny", 0), case.get("nz", 0)) or 2.0 * math.sqrt(C / max(1, case.get("count", 1)))
    if case["kind"] == "poisson":
        return dict(bytes=28 * K + (16 * F + 4 * W + 16) * C, flops=20.0 * K + 3.0 * side * (2 * W + 14.0) * C)
    n = {"solver": case.get("iters", 1), "piso": 1, "serve": 10}[case["kind"]]
    cg = 500 * 2 * max(1, case["refine"]) if case["kind"] == "piso" else 500 if case.get("channel") else min(500.0, 1.5 * side)
    return dict(bytes=n * (geometry + 2 * state + 2 * systems),
                flops=n * (200.0 * K + 100.0 * F * C + 3 * (12 * W + 90.0) * C + cg * (2 * W + 14.0) * C))


# ------------------------------------------------------------------- the same in 64 bits
# The loop cases run on a box of nx x ny x nz equal hexes, numbered i + nx (j + ny k); faces
# are numbered by their sorted node ids, which orders them by their lowest node and, at the
# same node, z before y before x.  A whole solver run has no such value: its pressure solves
# stop at a tolerance that leaves 32-bit and 64-bit runs apart by more than their rounding.
class _Box:
    def __init__(self, case):
        self.n = (case["nz"], case["ny"], case["nx"])   # array axes: z, y, x
        self.h = tuple(1.0 / s for s in self.n)
        self.V = self.h[0] * self.h[1] * self.h[2]
        self.A = tuple(self.V / h for h in self.h)

    def scatter(self, per_axis, width=None):
        """Face arrays (one per axis z, y, x, with one more plane than cells along it) in the
        mesh's face order."""
        nz, ny, nx = self.n
        node = torch.arange((nx + 1) * (ny + 1) * (nz + 1), device=DEVICE).reshape(nz + 1, ny + 1, nx + 1)
        keys, vals = [], []
        for a in range(3):
            cut = [slice(0, s + (1 if a == d else 0)) for d, s in enumerate(self.n)]
            keys.append((4 * node[tuple(cut)] + a).reshape(-1))
            vals.append(per_axis[a].reshape((-1,) if width is None else (-1, width)))
        order = torch.argsort(torch.cat(keys))
        return torch.cat(vals)[order]

    def gather(self, faces):
        """The inverse of scatter for a scalar per face."""
        sizes = [tuple(s + (1 if a == d else 0) for d, s in enumerate(self.n)) for a in range(3)]
        idx = [torch.arange(int(np.prod(s)), device=DEVICE, dtype=torch.int64) for s in sizes]
        for a in (1, 2):
            idx[a] = idx[a] + sum(int(np.prod(s)) for s in sizes[:a])
        order = self.scatter([i.reshape(s) for i, s in zip(idx, sizes)])
        flat = torch.empty(order.numel(), dtype=faces.dtype, device=DEVICE)
        flat[order] = faces
        out, at = [], 0
        for s in sizes:
            out.append(flat[at:at + int(np.prod(s))].reshape(s))
            at += int(np.prod(s))
        return out


def _ends(x, a, first, last):
    """x with one more plane before and after it along axis a."""
    return torch.cat([first, x, last], dim=a)


def _lo(x, a):
    return x.narrow(a, 0, 1)


def _hi(x, a):
    return x.narrow(a, x.shape[a] - 1, 1)


def _exact_fields(box, d):
    """Face values per axis (.., 4), fluxes per axis, gradients and divergence of the cavity."""
    phi = d["values"].double().reshape(*box.n, 4)
    fv, flux, grad = [], [], []
    for a in range(3):
        mid = 0.5 * (phi.narrow(a, 0, box.n[a] - 1) + phi.narrow(a, 1, box.n[a] - 1))
        wall = []
        for plane, lid in ((_lo(phi, a), False), (_hi(phi, a), a == 1)):
            w = torch.zeros_like(plane)
            w[..., 3] = plane[..., 3]
            if lid:
                w[..., 0] = float(np.float32(d["lid"]))
            wall.append(w)
        fv.append(_ends(mid, a, wall[0], wall[1]))
        flux.append(fv[a][..., 2 - a] * box.A[a])      # normal component: w, v, u for z, y, x
        grad.append((fv[a].narrow(a, 1, box.n[a]) - fv[a].narrow(a, 0, box.n[a])) / box.h[a])
    g = torch.stack([grad[2], grad[1], grad[0]], dim=-1)
    div = sum(flux[a].narrow(a, 1, box.n[a]) - flux[a].narrow(a, 0, box.n[a]) for a in range(3))
    return phi, fv, flux, g, div


def _outward(box, faces):
    """Fluxes as the mesh counts them: along its owner's outward normal.  The owner is the lower
    cell, so the first plane of each axis points the other way."""
    out = []
    for a in range(3):
        f = faces[a].clone()
        f.narrow(a, 0, 1).neg_()
        out.append(f)
    return out


def _apply(box, diag, lower, upper, x):
    """diag x + lower (towards smaller index) + upper (towards larger) per axis; x (.., m)."""
    y = diag * x
    for a in range(3):
        n = box.n[a]
        y.narrow(a, 1, n - 1).add_(lower[a].narrow(a, 1, n - 1).unsqueeze(-1) * x.narrow(a, 0, n - 1))
        y.narrow(a, 0, n - 1).add_(upper[a].narrow(a, 0, n - 1).unsqueeze(-1) * x.narrow(a, 1, n - 1))
    return y


def _exact_momentum(case, seed):
    box, d, c = _Box(case), _loop_inputs(case, seed), MOMENTUM
    phi, _, flux, g, _ = _exact_fields(box, d)
    nu, lid = float(np.float32(c["nu"])), float(np.float32(d["lid"]))
    diag = torch.full((*box.n, 3), box.V / c["dt"], dtype=torch.float64, device=DEVICE)
    rhs = phi[..., :3] * (box.V / c["dt"]) - g[..., 3, :] * (box.V / c["rho"])
    lower, upper = [], []
    for a in range(3):
        n, k = box.n[a], nu * box.A[a] / box.h[a]
        out_hi, out_lo = flux[a].narrow(a, 1, n), -flux[a].narrow(a, 0, n)
        lower.append(out_lo.clamp(max=0.0) - k)
        upper.append(out_hi.clamp(max=0.0) - k)
        diag += (out_hi.clamp(min=0.0) + out_lo.clamp(min=0.0) + 2 * k).unsqueeze(-1)
        for plane in (_lo(diag, a), _hi(diag, a)):     # walls: half a cell away, flux zero
            plane += k
        if a == 1:
            _hi(rhs, a)[..., 0] += 2 * k * lid
    al = c["relax"]
    rhs = rhs + (1 - al) / al * diag * phi[..., :3]
    diag = diag / al
    x = phi[..., :3].clone()                            # Jacobi: strongly diagonally dominant
    for _ in range(2000):
        r = rhs - _apply(box, diag, lower, upper, x)
        x = x + r / diag
        if float(r.norm()) < 1e-14 * float(rhs.norm()):
            break
    return dict(diag=diag.reshape(-1), rhs=rhs.reshape(-1), x=x.reshape(-1))


def _exact_poisson(case, seed):
    box, d = _Box(case), _loop_inputs(case, seed)
    k = box.gather(d["kappa"].double())
    diag = torch.zeros((*box.n, 1), dtype=torch.float64, device=DEVICE)
    lower, upper = [], []
    for a in range(3):
        n, f = box.n[a], k[a] * box.A[a] / box.h[a]
        f = f.clone()
        _lo(f, a).zero_()                               # walls of fixed gradient
        if a == 2:
            _hi(f, a).mul_(2.0)                         # the fixed value, half a cell away
        else:
            _hi(f, a).zero_()
        lower.append(f.narrow(a, 0, n))
        upper.append(f.narrow(a, 1, n))
        diag -= (lower[a] + upper[a]).unsqueeze(-1)
    rhs = d["source"].double().reshape(*box.n, 1)
    x, r = torch.zeros_like(rhs), rhs.clone()
    p, rz = torch.zeros_like(rhs), None
    for i in range(20000):
        z = r / diag
        new = float((r * z).sum())
        p = z + (new / rz if rz is not None else 0.0) * p
        rz = new
        q = _apply(box, diag, lower, upper, p)
        alpha = rz / float((p * q).sum())
        x, r = x + alpha * p, r - alpha * q
        if float(r.norm()) < 1e-13 * float(rhs.norm()):
            break
    return dict(diag=diag.reshape(-1), rhs=rhs.reshape(-1), x=x.reshape(-1))


def exact(case, seed):
    if case["kind"] == "fields":
        box, d = _Box(case), _loop_inputs(case, seed)
        _, fv, flux, g, div = _exact_fields(box, d)
        return dict(face_values=box.scatter(fv, 4), mass_fluxes=box.scatter(_outward(box, flux)),
                    cell_gradients=g.reshape(-1, 4, 3), div=div.reshape(-1))
    if case["kind"] == "momentum":
        return _exact_momentum(case, seed)
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    return None
