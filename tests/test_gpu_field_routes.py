"""The boundary tables applied by their own kernel are what the pass over every face writes."""
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
