"""The batched pressure CGs at the sizes where their kernels change: a case's bits are the same
alone (the kernel for its own rows per CTA) and beside a case that asks for the kernel of the
most rows per CTA."""
import numpy as np
import pytest
import torch

from tests.cases import cavity_bc, cavity_mesh, channel_bc, channel_mesh
from tests.gpu_helpers import fields, make_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300.build import build_library
    build_library()


def _cases(sizes):
    out = []
    for nx, ny in sizes:
        mesh, bc, ref = (cavity_mesh(nx), cavity_bc, 0) if nx == ny else (channel_mesh(nx, ny), channel_bc, None)
        out.append(make_pair(mesh, bc, ref_cell=ref, nu=0.02, u_relax=0.5)[:2])
    return out


# rows per CTA around 512, 1,024, 2,048 and up to 4,096 (one CTA a case, then four)
@pytest.mark.parametrize("cluster,sizes", [(1, [(8, 8), (22, 22), (23, 23), (32, 32), (33, 33), (45, 45), (46, 46), (64, 64)]),
                                           (4, [(32, 32), (90, 22), (91, 23), (90, 90), (92, 91), (128, 128)])])
@pytest.mark.parametrize("variant", [0, 1])
def test_bits_do_not_depend_on_the_batch(variant, cluster, sizes):
    from warpcfd_gb300.batch import CaseBatch

    mix = _cases(sizes)
    batch = CaseBatch([s for _, s in mix], cluster_size=cluster, cg_variant=variant)
    for _ in range(3):
        batch.step()
    got = [fields(m) for m, _ in mix]
    assert all(np.isfinite(g).all() for g in got)
    for i, (model, solver) in enumerate(_cases(sizes)):
        alone = CaseBatch([solver], cluster_size=cluster, cg_variant=variant)
        for _ in range(3):
            alone.step()
        assert np.array_equal(fields(model), got[i]), sizes[i]
