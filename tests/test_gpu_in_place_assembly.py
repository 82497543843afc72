"""Assembly with the off-diagonals in place (wcfd_mesh.slot_mask, the layout of structured meshes past
65,536 cells), on small meshes: every coefficient where its face's slot says, no stale padding, the
same diagonal, right-hand side, matrix and product as with the compact layout, and the oracle's."""
import itertools

import pytest
import torch

from tests.cases import (cavity3d_bc, cavity3d_mesh, cavity_bc, cavity_mesh, channel_bc, channel_mesh)
from tests.gpu_helpers import make_pair
from warpcfd_gb300.FV import geometry

pytestmark = pytest.mark.gpu

# mesh, boundary conditions, reference cell (inside, at a corner, none), slots that hold faces
MESHES = {
    "cavity": (lambda: cavity_mesh(9, jitter=0.15, seed=3), cavity_bc, 40, 0b111100),
    "channel": (lambda: channel_mesh(21, 5), channel_bc, None, 0b111100),
    "line": (lambda: channel_mesh(130, 1), channel_bc, 129, 0b101000),
    "hex": (lambda: cavity3d_mesh(6, jitter=0.1, seed=4), cavity3d_bc, 0, 0b111111),
}


@pytest.fixture(scope="module", autouse=True)
def _lib_ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300.build import build_library
    build_library()


def _solver(case, rows, monkeypatch, **kw):
    mk, bc, ref, mask = MESHES[case]
    monkeypatch.setattr(geometry, "CLUSTER_ROWS", rows)
    model, solver, _ = make_pair(mk(), bc, ref_cell=ref, **kw)
    assert (model._geo["slot_mask"] & 0xffff) == (0 if rows else mask)
    g = torch.Generator(device="cuda").manual_seed(8)
    for a in (model.cell_values, model.cell_gradients, model.face_values, model.face_gradients, model.mass_fluxes,
              solver.div_u):
        a.copy_(torch.randn(a.shape, generator=g, device="cuda"))
    solver.rUA_faces.copy_(0.1 + torch.rand(solver.rUA_faces.shape, generator=g, device="cuda"))
    return model, solver


def _compare(compact, placed):
    """compact, placed: Equations assembled in the two layouts; the coefficients of placed in face order."""
    assert torch.equal(compact.diag, placed.diag) and torch.equal(compact.rhs, placed.rhs)
    a, b = compact.matrix, placed.matrix
    assert torch.equal(a.col_indices(), b.col_indices()) and torch.equal(a.crow_indices(), b.crow_indices())
    assert torch.equal(a.values(), b.values())
    g = placed.fvm._geo
    C, W = g["n_cells"], g["ell_width"]
    own = g["ell_col"][:W] == torch.arange(C, device="cuda", dtype=torch.int32)
    off = placed.off[:W * C].reshape(W, C)
    assert bool((off[own] == 0).all()) and bool(torch.isfinite(off).all())
    x = torch.randn(placed.diag.shape, generator=torch.Generator(device="cuda").manual_seed(9), device="cuda")
    assert torch.equal(compact.apply(x), placed.apply(x))


def _stale(*equations):
    for e in equations:
        for a in (e.diag, e.off, e.rhs):
            a.fill_(float("nan"))


@pytest.mark.parametrize("case,scheme,explicit,steady",
                         [(c, s, x, t) for c, (s, x, t) in itertools.product(MESHES, [
                             ("upwind", False, True), ("upwind", True, False), ("upwindLinear", True, True),
                             ("central difference", False, True)])])
def test_momentum_and_pressure_systems(case, scheme, explicit, steady, monkeypatch):
    pair = []
    for rows in (65536, 0):
        _, s = _solver(case, rows, monkeypatch, steady=steady, dt=0.1, correction=explicit)
        s.convection.interpolation = scheme
        s.explicit_internal_terms = explicit
        _stale(s.vel_equation, s.p_corr_equation)
        s.assemble_momentum()
        s.assemble_pressure()
        pair.append(s)
    _compare(pair[0].vel_equation, pair[1].vel_equation)
    _compare(pair[0].p_corr_equation, pair[1].p_corr_equation)
    assert torch.equal(pair[0].rUA, pair[1].rUA)


@pytest.mark.parametrize("case", MESHES)
def test_systems_from_terms(case, monkeypatch):
    from warpcfd_gb300.FV.terms import ConvectionTerm, DdtTerm, DiffusionTerm, Equation, GradTerm
    vel, out = ["u", "v", "w"], []
    for rows in (65536, 0):
        model, s = _solver(case, rows, monkeypatch)
        t = [ConvectionTerm(model, vel, "central difference"), DiffusionTerm(model, vel), DdtTerm(model, vel),
             GradTerm(model, "p"), DiffusionTerm(model, "p")]
        t[0](model)
        t[1](model, viscosity=0.03)
        t[2](model, dt=0.1)
        t[3](model)
        t[4](model, viscosity=s.rUA_faces)
        v, p = Equation(model, vel), Equation(model, "p", solver="cg")
        _stale(v, p)
        v.form_system([t[0], -t[1], t[2]], explicit_terms=-1.0 * t[3])
        p.form_system(t[4])
        p.replace_row(model.num_cells // 2, 0.25)
        out.append((v, p))
    for compact, placed in zip(*out):
        _compare(compact, placed)


@pytest.mark.parametrize("case", ["cavity", "channel", "cavity3d"])
def test_assembly_matches_the_oracle(case, monkeypatch):
    from tests import test_gpu_parity, test_gpu_terms
    monkeypatch.setattr(geometry, "CLUSTER_ROWS", 0)
    test_gpu_parity.test_assembly_matches_oracle(case)
    for steady in (True, False):
        test_gpu_terms.test_form_system_from_terms_matches_oracle_assembly({"cavity": "cavity_corrected"}.get(case, case), steady)


@pytest.mark.parametrize("case", ["cavity_skew", "channel", "cavity3d"])
def test_steps_track_the_oracle(case, monkeypatch):
    """Whole steps on the grid kernels, which such meshes get."""
    from tests import test_gpu_parity
    from warpcfd_gb300 import _lib
    monkeypatch.setattr(geometry, "CLUSTER_ROWS", 0)
    _lib.call("wcfd_set_krylov_path", 1)
    try:
        test_gpu_parity.test_simple_steps_track_oracle(case)
    finally:
        _lib.call("wcfd_set_krylov_path", 0)
