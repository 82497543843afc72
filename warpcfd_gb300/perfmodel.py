"""Algorithmic (compulsory) HBM bytes of the kernels of one SIMPLE outer iteration.

Each array a kernel must touch is counted once per launch at its storage width (fp32
values, int32 indices, float4-packed geometry).  Gathers of neighbour values that a
kernel already streams elsewhere are not counted again.  C cells, K faces (Ki internal,
B boundary), F slots per cell, W off-diagonal width, k Krylov iterations.
"""
from __future__ import annotations


def cg_bytes_per_iteration(C: int, W: int, col_bytes: int = 4) -> int:
    """One CG iteration (two passes) per row, r, q, x and 1/diag held in shared memory:
    p = z + beta p_old ; q = A p : off 4W + col (col_bytes) W + diag 4 + z 4 + p_old 4 + p 4 (w)
    r -= alpha q ; z = M r       : z 4 (w)
    col_bytes 2 when the columns are read as int16 offsets (wcfd_mesh.ell_dcol), 0 when the
    off-diagonals stand in place (wcfd_mesh.slot_mask) and a chunk of rows shares its offsets.
    """
    return C * ((4 + col_bytes) * W + 20)


def cg_bytes_setup(C: int, W: int, col_bytes: int = 4) -> int:
    """r = b - A x, invd, z, p: off/col (4 + col_bytes) W, diag 4, x 4, b 4, writes r, invd, z, p 16."""
    return C * ((4 + col_bytes) * W + 28)


def cg_bytes(C: int, W: int, iters: int, col_bytes: int = 4) -> int:
    return cg_bytes_setup(C, W, col_bytes) + iters * cg_bytes_per_iteration(C, W, col_bytes)


BICG_BLOCKS, BICG_ROWS_PER_BLOCK = 152, 256  # most blocks of the grid BiCGSTAB, rows it gives a block before that
BICG_BLOCK_BYTES = 232448 - 4176             # a block's shared memory, less what the kernel itself takes


def bicgstab_resident(C: int, W: int) -> bool:
    """Whether the grid BiCGSTAB keeps a block's rows in shared memory (launch_krylov, capi.cu): rows per
    block rounded up to 32, 24 + 2 W floats a row."""
    blocks = max(1, min(BICG_BLOCKS, -(-C // BICG_ROWS_PER_BLOCK)))
    rows = -(-(-(-C // blocks)) // 32) * 32
    return rows * (96 + 8 * W) <= BICG_BLOCK_BYTES


def bicgstab_bytes_per_iteration(C: int, W: int, col_bytes: int = 4) -> int:
    """One BiCGSTAB iteration on the 3-component system, per cell; records R = (r, 1/d_0),
    U = (u, 1/d_1), V = (v, 1/d_1) of 16 B and Z = 1/d_2 of 4 B:
    v = A M p : R, U, Z 36 + V 16 (w)
    t = A M s : R, V, Z 36
    x, r, u   : R, U 32 (w)
    A resident system moves those; a streamed one also off/col (4 + col_bytes) W + diag 12 in
    each product, r0 12 + p 12 (w), t 12 (w), and R, V, Z 36 + r0, p, t, x 48 + x 12 (w).
    """
    if bicgstab_resident(C, W):
        return C * 120
    return C * (2 * (4 + col_bytes) * W + 276)


def bicgstab_bytes(C: int, W: int, iters: int, col_bytes: int = 4) -> int:
    setup = C * (8 * W + 12 + 12 + 12 + 12 * 4)
    return setup + iters * bicgstab_bytes_per_iteration(C, W, col_bytes)


def face_pass_bytes(C: int, K: int, Ki: int, B: int, mdot: bool = True) -> int:
    """Every field: internal faces only write their values (16), boundary faces read and
    write them (32) and their gradients."""
    b = 8 * K + 16 * Ki + 16 * K + 16 * B + 64 * C  # owner/nbr, interp, face values, cell values+grads
    b += B * (4 + 4 + 16 + 32 + 4)                   # brow, bc type, bc value, face grads rw, rpf
    if mdot:
        b += 16 * K + 4 * K
    return b


def face_pass_partial_bytes(C: int, K: int, Ki: int, B: int) -> int:
    """One field (the pressure-only pass, no mass flux): face records read and written
    whole (32), the cells' value records (16) and the field's 3 gradient components (12)."""
    return 8 * K + 16 * Ki + 32 * K + 28 * C + B * (4 + 4 + 16 + 16 + 4)


def gradient_bytes(C: int, K: int, F: int, div: bool = False) -> int:
    b = 16 * F * C + 16 * K + 48 * C
    if div:
        b += 4 * K + 4 * C
    return b


def momentum_assembly_bytes(C: int, K: int, F: int, W: int, B: int) -> int:
    return (16 * F * C + 4 * K + 4 * K + 4 * K + B * (4 + 4 + 16 + 16 + 4) + 4 * W * C + 24 * C + 16 * C + 48 * C
            + 4 * C + 4 * C)


def pressure_assembly_bytes(C: int, K: int, F: int, W: int, B: int) -> int:
    return 16 * F * C + 4 * K + 4 * K + 4 * K + B * (4 + 1 + 8) + 4 * W * C + 8 * C + 4 * C


def simple_step_bytes(C, K, Ki, B, F, W, k_u, k_p, n_corr=1, col_bytes=4) -> dict:
    d = {
        "face_pass": face_pass_bytes(C, K, Ki, B) * 2 * n_corr + face_pass_bytes(C, K, Ki, B, mdot=False) * n_corr,
        "gradient": gradient_bytes(C, K, F) + gradient_bytes(C, K, F, div=True) * n_corr
        + gradient_bytes(C, K, F) * n_corr,
        "momentum_assemble": momentum_assembly_bytes(C, K, F, W, B),
        "pressure_assemble": pressure_assembly_bytes(C, K, F, W, B) * n_corr,
        "bicgstab": bicgstab_bytes(C, W, k_u, max(col_bytes, 2)),
        "cg": cg_bytes(C, W, k_p, col_bytes) * n_corr,
        "small": 32 * C + 12 * K,
    }
    d["total"] = sum(d.values())
    return d
