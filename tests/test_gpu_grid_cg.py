"""The grid CG on the same box operator in its layouts: off-diagonals in place, from slot 0 on,
and with the rows renumbered at random (no chunk of rows with common column offsets), at sizes
around its chunks, blocks and shared memory."""
import ctypes as ct

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _grid_path():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300 import _lib
    from warpcfd_gb300.build import build_library
    build_library()
    _lib.call("wcfd_set_krylov_path", 1)
    yield
    _lib.call("wcfd_set_krylov_path", 0)


def _box(n, seed=0):
    """(columns, coefficients, diagonal, right-hand side) of a variable-coefficient 7-point
    operator on an nx x ny x nz box, slots -z, +z, -y, +x, +y, -x as a hex mesh has them, in
    place; axes of one cell have no slots."""
    nx, ny, nz = n
    C = nx * ny * nz
    g = torch.Generator(device="cuda").manual_seed(seed)
    idx = torch.arange(C, device="cuda").reshape(nz, ny, nx)
    cols, offs = [], []
    for axis, up, size in ((0, False, nz), (0, True, nz), (1, False, ny), (2, True, nx), (1, True, ny), (2, False, nx)):
        if size == 1:
            continue
        k = 0.5 + torch.rand((nz, ny, nx), generator=torch.Generator(device="cuda").manual_seed(seed + axis),
                             device="cuda")               # coefficient of the face above each cell
        c, o = idx.clone(), torch.zeros((nz, ny, nx), device="cuda")
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[axis], hi[axis] = slice(0, size - 1), slice(1, size)
        if up:
            c[tuple(lo)], o[tuple(lo)] = idx[tuple(hi)], k[tuple(lo)]
        else:
            c[tuple(hi)], o[tuple(hi)] = idx[tuple(lo)], k[tuple(lo)]
        cols.append(c.reshape(-1))
        offs.append(o.reshape(-1))
    col, off = torch.stack(cols).int(), torch.stack(offs)
    diag = -(off.sum(0) + 0.01 + 0.1 * torch.rand(C, generator=g, device="cuda"))
    return col, off, diag, torch.randn(C, generator=g, device="cuda")


def _compact(col, off):
    C = col.shape[1]
    own = torch.arange(C, device="cuda", dtype=torch.int32)
    order = torch.argsort((col == own).int(), dim=0, stable=True)
    return torch.gather(col, 0, order).contiguous(), torch.gather(off, 0, order).contiguous()


def _solve(col, off, diag, rhs, mask=0, offsets=False, maxiter=60, atol=0.0):
    from warpcfd_gb300 import _lib
    W, C = col.shape
    col, off = col.contiguous(), off.contiguous()
    d16 = (col - torch.arange(C, device="cuda", dtype=torch.int32)).to(torch.int16) if offsets else None
    dummy = torch.zeros(8, device="cuda").data_ptr()
    m = _lib.Mesh_t()
    m.n_cells, m.n_faces, m.faces_per_cell, m.ell_width = C, 1, 6, W
    m.slot_mask = _lib.SLOT_MASK | mask if mask else 0
    for name in ("face_owner", "face_nbr", "face_brow", "face_interp", "face_normal", "face_gdiff", "face_rpf",
                 "cell_slot", "cell_volume"):
        setattr(m, name, dummy)
    m.ell_col = col.data_ptr()
    m.ell_dcol = d16.data_ptr() if offsets else None
    x = torch.zeros(C, device="cuda")
    ws = torch.full((int(_lib.load().wcfd_krylov_workspace_floats(C, 1)),), float("nan"), device="cuda")
    part = torch.zeros(8 * _lib.MAX_BLOCKS, dtype=torch.float64, device="cuda")
    bar = torch.zeros(_lib.BARRIER_WORDS, dtype=torch.int32, device="cuda")
    stats = torch.zeros(_lib.STATS_BYTES, dtype=torch.uint8, device="cuda")
    A = _lib.System_t(diag.data_ptr(), off.data_ptr(), rhs.data_ptr(), 1, 0)
    w = _lib.KrylovWS_t(ws.data_ptr(), part.data_ptr(), None, bar.data_ptr())
    _lib.call("wcfd_cg", ct.byref(m), A, ct.c_void_p(x.data_ptr()), w, atol, maxiter, ct.c_void_p(stats.data_ptr()),
              ct.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return x, np.frombuffer(stats.cpu().numpy().tobytes(), dtype=_lib.STATS_DTYPE)[0]


def _residual(col, off, diag, rhs, x):
    r = rhs.double() - diag.double() * x.double()
    for j in range(col.shape[0]):
        r -= off[j].double() * x.double()[col[j].long()]
    return float(r.norm())


# chunk edges (32 to 128 rows), one and several blocks, 1 to 4 rows of a thread and more,
# two-, four- and six-slot rows
@pytest.mark.parametrize("n,mask", [((31, 1, 1), 0b101000), ((33, 2, 1), 0b111100), ((16, 16, 2), 0b111111),
                                    ((129, 9, 7), 0b111111), ((61, 47, 53), 0b111111), ((346, 346, 1), 0b111100),
                                    ((70, 60, 55), 0b111111), ((67, 66, 65), 0b111111), ((96, 90, 100), 0b111111)])
def test_layouts_give_the_same_bits(n, mask):
    col, off, diag, rhs = _box(n)
    cc, oc = _compact(col, off)
    want, st = _solve(cc, oc, diag, rhs)
    assert st["iterations"] == 60 or st["status"] == 3 or st["residual"] < 1e-10   # a short row may end early
    for offsets in (False, True):
        if offsets and int((col - torch.arange(col.shape[1], device="cuda")).abs().max()) > 32767:
            continue
        got, s2 = _solve(col, off, diag, rhs, mask, offsets)
        assert torch.equal(got, want) and s2 == st, offsets
        assert torch.equal(_solve(cc, oc, diag, rhs, 0, offsets)[0], want), offsets
    # a renumbered system has no regular chunk: the same solution to the solve's tolerance.
    # Both run to ||r|| <= 1e-3; diag dominance >= 0.01 bounds each error by 1e-3 / 0.01 in the
    # 2-norm
    C = col.shape[1]
    perm = torch.randperm(C, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    inv = torch.empty_like(perm)
    inv[perm] = torch.arange(C, device="cuda")
    pc, po = inv[cc.long()][:, perm].int(), oc[:, perm]
    a, sa = _solve(cc, oc, diag, rhs, maxiter=500, atol=1e-3)
    p, sp = _solve(pc, po, diag[perm].contiguous(), rhs[perm].contiguous(), maxiter=500, atol=1e-3)
    assert sa["status"] == 0 and sp["status"] == 0
    assert float((p[inv].double() - a.double()).norm()) <= 2 * 1e-3 / 0.01


def test_rows_past_shared_memory_and_coefficients_on_padding():
    """More rows per block than shared memory holds, and a caller's matrix with coefficients on
    padding slots (they act on the row itself): the reported residual is that of the solution."""
    col, off, diag, rhs = _box((190, 160, 120))        # 24,000 rows a block
    x, st = _solve(col, off, diag, rhs, 0b111111, maxiter=400, atol=1e-2)
    assert st["status"] == 0
    r = _residual(col, off, diag, rhs, x)
    # the recurrence's residual and the true one part by rounding: eps times the sum of
    # |A||x| over the iterations, here < 400 * 6e-8 * ||A|| ||x||
    bound = 400 * 6e-8 * 14.0 * float(x.double().norm())
    assert abs(r - st["residual"]) <= bound and st["residual"] <= 1e-2
    y, _ = _solve(*_compact(col, off), diag, rhs, maxiter=400, atol=1e-2)
    assert torch.equal(x, y)
    col, off, diag, rhs = _box((40, 30, 20), seed=5)
    own = torch.arange(col.shape[1], device="cuda", dtype=torch.int32)
    off = torch.where(col == own, torch.full_like(off, -0.25), off)
    x, st = _solve(col, off, diag, rhs, 0b111111, maxiter=500, atol=1e-3)
    r = _residual(col, off, diag, rhs, x)
    assert st["status"] == 0 and abs(r - st["residual"]) <= 500 * 6e-8 * 14.0 * float(x.double().norm())


# one CTA to sixteen, 1 to 8 rows of a thread and ragged last CTAs, around the cluster CG's
# 512, 1,024 and 2,048 rows per CTA
@pytest.mark.parametrize("n", [(7, 1, 1), (64, 8, 1), (129, 4, 1), (91, 90, 1), (100, 164, 1), (181, 181, 1), (205, 160, 1),
                               (26, 25, 24), (32, 32, 32), (33, 32, 32)])
def test_cluster_solve_matches_the_grid_solve(n):
    """Both solve to ||r|| <= 1e-3; diagonal dominance >= 0.01 bounds each error by 1e-3 / 0.01.
    The reported residual norms are those of the solutions up to the recurrence's rounding (see
    above)."""
    from warpcfd_gb300 import _lib
    cc, oc = _compact(*_box(n)[:2])
    _, _, diag, rhs = _box(n)
    a, sa = _solve(cc, oc, diag, rhs, maxiter=500, atol=1e-3)
    _lib.call("wcfd_set_krylov_path", 2)
    try:
        b, sb = _solve(cc, oc, diag, rhs, maxiter=500, atol=1e-3)
        c, sc = _solve(cc, oc, diag, rhs, maxiter=500, atol=1e-3)
    finally:
        _lib.call("wcfd_set_krylov_path", 1)
    assert sa["status"] == 0 and sb["status"] == 0
    assert torch.equal(b, c) and sb == sc
    assert float((a.double() - b.double()).norm()) <= 2 * 1e-3 / 0.01
    bound = 500 * 6e-8 * 14.0 * float(b.double().norm())
    assert abs(_residual(cc, oc, diag, rhs, b) - sb["residual"]) <= bound
    assert abs(sb["rhs_norm"] - float(rhs.double().norm())) <= 1e-6 * sb["rhs_norm"]
