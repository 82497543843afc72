"""The boundary tables applied by their own kernel are what the pass over every face writes; term
weights and their assembly at the edges of their blocks (128 cells, 256 slots) and from arrays
that are not 16-byte aligned."""
import ctypes as ct

import pytest
import torch

from tests.cases import cavity_bc, cavity_mesh, channel_bc, channel_mesh
from tests.gpu_helpers import make_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300.build import build_library
    build_library()


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 7), (16, 16), (63, 65), (130, 3)])
def test_boundary_values(nx, ny):
    from warpcfd_gb300 import _lib

    mesh, bc, ref = (cavity_mesh(nx), cavity_bc, 0) if nx == ny else (channel_mesh(nx, ny), channel_bc, None)
    model = make_pair(mesh, bc, ref_cell=ref, nu=0.02, u_relax=0.5)[0]
    g = torch.Generator(device="cuda").manual_seed(nx * 1000 + ny)
    start = [torch.randn(a.shape, generator=g, device="cuda") for a in (model.face_values, model.face_gradients)]
    arrays = (model.face_values, model.face_gradients)
    out = []
    for own in (True, False):
        for a, b in zip(arrays, start):
            a.copy_(b)
        if own:
            model.set_boundary_conditions()
        else:
            _lib.call("wcfd_face_pass_flags", ct.byref(model.mesh_struct()), model.bc_struct(), model.state_struct(), 0, 1,
                      ct.c_void_p(torch.cuda.current_stream().cuda_stream))
        out.append([a.clone() for a in arrays])
    assert not torch.equal(out[0][0], start[0]) or not torch.equal(out[0][1], start[1])
    for a, b in zip(*out):
        assert torch.equal(a, b)


# 127 to 129 cells and several blocks; six slots a cell
@pytest.mark.parametrize("nx,ny", [(127, 1), (64, 2), (43, 3), (86, 6)])
def test_term_blocks_match_the_oracle(nx, ny, monkeypatch):
    from tests import test_gpu_terms as terms

    monkeypatch.setitem(terms.CASES, "blocks", (lambda: channel_mesh(nx, ny), channel_bc, None, False))
    terms.test_term_weights_match_oracle("blocks")


@pytest.mark.parametrize("nx,ny", [(127, 1), (64, 2), (43, 3), (86, 6)])
def test_assembly_does_not_depend_on_alignment(nx, ny):
    """Each off-diagonal and diagonal is the sum of its weights in term order: the same bits from
    aligned and shifted arrays, and as a plain loop over the slots gives (fp64, within the fp32
    rounding of at most 13 additions, 13 * 6e-8 of the sum of magnitudes)."""
    from warpcfd_gb300 import _lib
    from warpcfd_gb300.FV.terms import ConvectionTerm, DdtTerm, DiffusionTerm, Equation

    model = make_pair(channel_mesh(nx, ny), channel_bc, nu=0.02, u_relax=0.5)[0]
    g = torch.Generator(device="cuda").manual_seed(nx)
    model.cell_values.copy_(torch.randn(model.cell_values.shape, generator=g, device="cuda"))
    model.set_boundary_conditions()
    model.face_interpolation()
    model.calculate_mass_flux()
    model.calculate_gradients()
    vel = ["u", "v", "w"]
    t = [ConvectionTerm(model, vel, "upwind"), DiffusionTerm(model, vel), DdtTerm(model, vel)]
    t[0](model)
    t[1](model, viscosity=0.03)
    t[2](model, dt=0.1)
    eq = Equation(model, vel)
    eq.form_system([t[0], -t[1], t[2]])
    want = [a.clone() for a in (eq.diag, eq.off, eq.rhs)]
    arr = (_lib.Term_t * 3)()
    keep = []
    for i, (term, sc) in enumerate(zip(t, (1.0, -1.0, 1.0))):
        n = term.weights.numel()
        buf = torch.zeros(n + 4, device="cuda")
        buf[1:n + 1].copy_(term.weights.reshape(-1))
        keep.append(buf)
        arr[i].weights, arr[i].scale, arr[i].cell_based = buf.data_ptr() + 4, sc, int(term.cell_based)
    for a in (eq.diag, eq.off, eq.rhs):
        a.fill_(float("nan"))
    _lib.call("wcfd_assemble_terms", ct.byref(model.mesh_struct()), eq.system_struct(), arr, 3,
              ct.c_void_p(torch.cuda.current_stream().cuda_stream))
    for a, b in zip((eq.diag, eq.off, eq.rhs), want):
        assert torch.equal(a, b)
    w0, w1, w2 = (x.weights.double() for x in t)
    diag = w0[..., 0].sum(1) - w1[..., 0].sum(1) + w2[..., 0]
    size = w0[..., 0].abs().sum(1) + w1[..., 0].abs().sum(1) + w2[..., 0].abs()
    assert ((want[0].double().reshape(-1, 3) - diag).abs() <= 13 * 6e-8 * size).all()
