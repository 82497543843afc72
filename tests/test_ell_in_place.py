"""Off-diagonals in place (wcfd_mesh.slot_mask): chosen for large structured numberings only;
every used face slot then has its own off-diagonal slot, boundary faces as padding, and the
columns of a row are those of the compact layout in the same order."""
import numpy as np
import pytest

from warpcfd_gb300._lib import SLOT_MASK
from warpcfd_gb300.FV import geometry
from warpcfd_gb300.preprocess import Mesh, create_2D_grid, create_3D_grid


def _mesh(kind, n):
    if kind == "2d":
        return Mesh(create_2D_grid((0, 0, 0), *n, 1.0, 1.0, 0.1))
    return Mesh(create_3D_grid((0, 0, 0), *n, 1.0, 1.0, 1.0, element_type="tetra" if kind == "tetra" else "hex"))


@pytest.mark.parametrize("kind,n,mask", [("2d", (9, 7), 0b111100), ("hex", (5, 4, 3), 0b111111), ("tetra", (3, 2, 2), 0),
                                         ("2d", (9, 1), 0b101000), ("2d", (1, 1), 0)])
def test_in_place_layout(monkeypatch, kind, n, mask):
    m = _mesh(kind, n)
    compact = geometry.build_geometry(m)
    assert compact["slot_mask"] == 0          # below the cluster solvers' reach
    monkeypatch.setattr(geometry, "CLUSTER_ROWS", 0)
    g = geometry.build_geometry(m)
    assert g["slot_mask"] == (SLOT_MASK | mask if mask else 0)
    C, W = g["n_cells"], g["ell_width"]
    assert W == compact["ell_width"]
    slots = [f for f in range(g["faces_per_cell"]) if mask >> f & 1]
    nbr = m.cell_properties.neighbors
    for c in range(C):
        row = g["ell_col"][:W, c]
        assert [v for v in row if v != c] == [v for v in compact["ell_col"][:W, c] if v != c]
        if mask:
            assert list(row) == [nbr[c, f] if nbr[c, f] >= 0 else c for f in slots]
    if W:
        rows = np.arange(C)[None, :]
        assert np.array_equal(g["ell_dcol"].astype(np.int64) + rows, g["ell_col"].astype(np.int64))
