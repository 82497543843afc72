"""The byte model follows the launcher's rule for the resident grid BiCGSTAB: 152 blocks, rows rounded up to
32, 96 + 8 W bytes of shared memory a row beside 4,176 of the kernel's own."""
import pytest

from warpcfd_gb300 import perfmodel


@pytest.mark.parametrize("W,last", [(6, 152 * 1568), (5, 152 * 1664), (4, 152 * 1760), (0, 152 * 2368)])
def test_resident_limit(W, last):
    assert last // 152 * (96 + 8 * W) <= 232448 - 4176 < (last // 152 + 32) * (96 + 8 * W)
    assert perfmodel.bicgstab_resident(last, W) and not perfmodel.bicgstab_resident(last + 1, W)
    assert perfmodel.bicgstab_resident(1, W)
    assert perfmodel.bicgstab_bytes_per_iteration(last, W) == last * 120
    assert perfmodel.bicgstab_bytes_per_iteration(last + 1, W) > last * 200
