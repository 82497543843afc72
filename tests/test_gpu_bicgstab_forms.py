"""The BiCGSTAB in its forms -- over one cluster, over the grid with a block's rows in shared memory,
over the grid with the matrix streamed -- on a box operator with three diagonals, at the sizes
where they change."""
import ctypes as ct

import numpy as np
import pytest
import torch

from tests.test_gpu_grid_cg import _box, _compact

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300 import _lib
    from warpcfd_gb300.build import build_library
    build_library()
    yield
    _lib.call("wcfd_set_krylov_path", 0)


def _solve(col, off, diag, rhs, mask=0, offsets=False, path=0, shift=0):
    """shift: floats by which the workspace misses 16-byte alignment."""
    from warpcfd_gb300 import _lib
    W, C = col.shape
    col, off = col.contiguous(), off.contiguous()
    d16 = (col - torch.arange(C, device="cuda", dtype=torch.int32)).to(torch.int16) if offsets else None
    spare = torch.zeros(8, device="cuda")
    dummy = spare.data_ptr()
    m = _lib.Mesh_t()
    m.n_cells, m.n_faces, m.faces_per_cell, m.ell_width = C, 1, 6, W
    m.slot_mask = _lib.SLOT_MASK | mask if mask else 0
    for name in ("face_owner", "face_nbr", "face_brow", "face_interp", "face_normal", "face_gdiff", "face_rpf",
                 "cell_slot", "cell_volume"):
        setattr(m, name, dummy)
    m.ell_col = col.data_ptr() or dummy
    m.ell_dcol = (d16.data_ptr() or dummy) if offsets else None
    x = torch.zeros(3 * C, device="cuda")
    n = int(_lib.load().wcfd_krylov_workspace_floats(C, 3))
    ws = torch.full((n + 64,), float("nan"), device="cuda")
    part = torch.zeros(8 * _lib.MAX_BLOCKS, dtype=torch.float64, device="cuda")
    bar = torch.zeros(_lib.BARRIER_WORDS, dtype=torch.int32, device="cuda")
    stats = torch.zeros(_lib.STATS_BYTES, dtype=torch.uint8, device="cuda")
    A = _lib.System_t(diag.data_ptr(), off.data_ptr() or dummy, rhs.data_ptr(), 3, 0)
    w = _lib.KrylovWS_t(ws.data_ptr() + 4 * shift, part.data_ptr(), None, bar.data_ptr())
    _lib.call("wcfd_set_krylov_path", path)
    _lib.call("wcfd_bicgstab", ct.byref(m), A, ct.c_void_p(x.data_ptr()), w, 1e-3, 500, ct.c_void_p(stats.data_ptr()),
              ct.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.isnan(ws[n + shift:]).all() and torch.isnan(ws[:shift]).all()
    return x, np.frombuffer(stats.cpu().numpy().tobytes(), dtype=_lib.STATS_DTYPE)[0]


def _residual(col, off, diag, rhs, x):
    x = x.double().reshape(-1, 3)
    r = rhs.double().reshape(-1, 3) - diag.double().reshape(-1, 3) * x
    for j in range(col.shape[0]):
        r -= off[j].double()[:, None] * x[col[j].long()]
    return float(r.norm())


# one row; around a CTA's 256 rows and 512 threads; the cluster's last size (16 x 1,033 rows of six
# slots) and the grid's first; the last rows that shared memory holds (about 152 x 1,600) and past it
@pytest.mark.parametrize("n,mask", [((1, 1, 1), 0), ((2, 1, 1), 0b101000), ((17, 15, 1), 0b111100), ((257, 1, 1), 0b101000),
                                    ((64, 64, 1), 0b111100), ((32, 16, 32), 0b111111), ((33, 16, 32), 0b111111),
                                    ((61, 47, 53), 0b111111), ((60, 60, 66), 0b111111), ((61, 60, 70), 0b111111)])
def test_forms_agree(n, mask):
    """Each form solves to ||r|| <= 1e-3 and reports the residual norm of its solution up to the
    recurrence's rounding (< 500 * 6e-8 * ||A|| ||x||, as for the CG); diagonal dominance >= 0.01
    bounds each error by 1e-3 / 0.01.  Layouts, column types and alignment do not show in a
    form's bits."""
    if n == (1, 1, 1):
        col, off = torch.zeros((0, 1), dtype=torch.int32, device="cuda"), torch.zeros((0, 1), device="cuda")
        diag, rhs = torch.tensor([-2.0], device="cuda"), torch.tensor([1.0], device="cuda")
    else:
        col, off, diag, rhs = _box(n)
    C = col.shape[1]
    g = torch.Generator(device="cuda").manual_seed(C)
    diag = (diag[:, None] * (1.0 + 0.2 * torch.rand((C, 3), generator=g, device="cuda"))).reshape(-1).contiguous()
    rhs = torch.randn(3 * C, generator=g, device="cuda")
    cc, oc = _compact(col, off) if col.shape[0] else (col, off)
    near = not col.shape[0] or int((col - torch.arange(C, device="cuda")).abs().max()) <= 32767
    xs = []
    for path in (1, 0):
        x, st = _solve(cc, oc, diag, rhs, path=path)
        # a single row is solved by its diagonal: s = 0 ends the iteration as a breakdown (omega = 0)
        assert st["status"] == (0 if C > 1 else 3) and st["residual"] <= 1e-3
        r = _residual(cc, oc, diag, rhs, x)
        assert abs(r - st["residual"]) <= 500 * 6e-8 * 14.0 * 1.2 * float(x.double().norm())
        assert abs(st["rhs_norm"] - float(rhs.double().norm())) <= 1e-6 * st["rhs_norm"]
        for kw in [dict(shift=1), dict(offsets=near)] + ([dict(mask=mask)] if mask else []):
            c, o = (col, off) if "mask" in kw else (cc, oc)
            y, s2 = _solve(c, o, diag, rhs, path=path, **kw)
            assert torch.equal(x, y) and s2 == st, (path, kw)
        xs.append(x.double())
    assert float((xs[0] - xs[1]).norm()) <= 2 * 1e-3 / 0.01
