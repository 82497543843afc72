"""Mesh arrays that name places to write: wcfd_check_mesh counts the entries that do not fit the rest of
the mesh, and kernels given such a mesh stay inside their arrays."""
import ctypes as ct

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300.build import build_library
    build_library()


def _check(mesh_struct):
    from warpcfd_gb300 import _lib
    out = (ct.c_int32 * 5)()
    return _lib.load().wcfd_check_mesh(ct.byref(mesh_struct), out, None), list(out)


def _in_place(monkeypatch, mesh, **kw):
    from tests.cases import cavity_bc
    from tests.gpu_helpers import make_pair
    from warpcfd_gb300.FV import geometry
    monkeypatch.setattr(geometry, "CLUSTER_ROWS", 0)
    model, solver, _ = make_pair(mesh, cavity_bc, **kw)
    assert model._geo["slot_mask"]
    return model, solver


def test_slot_mask_is_checked(monkeypatch):
    from tests.cases import cavity_mesh
    from warpcfd_gb300 import _lib
    model, _ = _in_place(monkeypatch, cavity_mesh(6))
    assert model.check_mesh() == [0] * 5
    C = model.num_cells
    internal = model._geo["face_nbr"].ge(0).sum().item()
    ms = model.mesh_struct()
    for mask in (0b001111, 0b111010):                  # as many slots, not the ones that hold the faces
        ms.slot_mask = _lib.SLOT_MASK | mask
        rc, c = _check(ms)
        assert rc == _lib.WCFD_ERR_ARGUMENT and c[:4] == [0] * 4 and c[4] >= internal / 2
    for mask in (0b011100, 0b1111000):                 # too few, and a slot that cells do not have
        ms.slot_mask = _lib.SLOT_MASK | mask
        with pytest.raises(_lib.WcfdError):
            _lib.check(_check(ms)[0])
    ms = model.mesh_struct()
    col = model._geo["ell_col"].clone()
    col[[0, 1]] = col[[1, 0]]                          # two slots' columns exchanged: every cell has one of them
    ms.ell_col = col.data_ptr()
    ms.ell_dcol = None
    rc, c = _check(ms)
    assert rc == _lib.WCFD_ERR_ARGUMENT and c[4] >= C


@pytest.mark.parametrize("what", ["momentum", "pressure"])
def test_assembly_with_a_wrong_slot_mask_stays_in_its_array(monkeypatch, what):
    """A mask that leaves faces of the last slots without an off-diagonal: nothing is written past
    the W * C coefficients."""
    from tests.cases import cavity_mesh
    from warpcfd_gb300 import _lib
    model, solver = _in_place(monkeypatch, cavity_mesh(6))
    solver.step()
    C, W = model.num_cells, model._geo["ell_width"]
    cs = _lib.Case_t.from_buffer_copy(solver.case_struct())
    cs.mesh.slot_mask = _lib.SLOT_MASK | 0b001111
    off = torch.full(((W + 2) * C,), 7.0, device="cuda")
    (cs.mom if what == "momentum" else cs.pres).off = off.data_ptr()
    _lib.call(f"wcfd_assemble_{what}", ct.byref(cs), None)
    torch.cuda.synchronize()
    assert bool((off[W * C:] == 7.0).all())
    assert np.isfinite(off.cpu().numpy()).all()


def test_boundary_list_is_checked_and_its_order_does_not_matter():
    """set_boundary_conditions goes by the list of boundary faces: entries that are no boundary face are
    counted and skipped, and every face gets its own row's values in whatever order the list has them."""
    from tests.cases import cavity_bc, cavity_mesh
    from tests.gpu_helpers import make_pair
    from warpcfd_gb300 import _lib
    model = make_pair(cavity_mesh(9), cavity_bc)[0]
    faces, K = model._geo["boundary_face"], model._geo["n_faces"]
    start = [torch.randn_like(a) for a in (model.face_values, model.face_gradients)]

    def apply(lst):
        ms = model.mesh_struct()
        ms.boundary_face = lst.data_ptr()
        for a, b in zip((model.face_values, model.face_gradients), start):
            a.copy_(b)
        _lib.call("wcfd_set_boundary_conditions", ct.byref(ms), model.bc_struct(), model.state_struct(), None)
        torch.cuda.synchronize()
        return _check(ms), model.face_values.clone(), model.face_gradients.clone()

    (rc, c), fv, fg = apply(faces)
    assert rc == 0 and c == [0] * 5 and not torch.equal(fv, start[0])
    (rc, c), fv2, fg2 = apply(faces.flip(0).contiguous())
    assert rc == _lib.WCFD_ERR_ARGUMENT and c[1] >= len(faces) - 1 and c[0] + c[2] + c[3] + c[4] == 0
    assert torch.equal(fv, fv2) and torch.equal(fg, fg2)
    bad = faces.clone()
    gone = bad[[0, 3, 5]].long()
    bad[0], bad[3], bad[5] = -1, K, int((model._geo["face_nbr"] >= 0).nonzero()[0])   # the last an internal face
    (rc, c), fv3, fg3 = apply(bad)
    assert rc == _lib.WCFD_ERR_ARGUMENT and c[1] == 3
    fv[gone], fg[gone] = start[0][gone], start[1][gone]
    assert torch.equal(fv, fv3) and torch.equal(fg, fg3)
