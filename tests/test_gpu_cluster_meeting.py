"""Meetings of a thread-block cluster (cluster_reduce): exact sums, and waits that run out.  A CTA that
leaves or comes late makes the others' bounded waits give up; every thread of a CTA takes the same
answer, every CTA returns and the context stays usable."""
import ctypes as ct

import pytest
import torch

pytestmark = pytest.mark.gpu
TIMEOUT = 5
# the CG's two, the BiCGSTAB's, the batched CG's two
FORMS = [(256, 1), (512, 1), (512, 0), (256, 2), (512, 2)]


@pytest.fixture(scope="module", autouse=True)
def _lib_ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from warpcfd_gb300.build import build_library
    build_library()


def _check(ctas, form, reductions, who=-1, at=0, delay_us=0, limit_us=200_000):
    from warpcfd_gb300 import _lib
    res = (ct.c_int32 * 16)()
    _lib.call("wcfd_cluster_meeting_check", ctas, form[0], form[1], reductions, who, at, int(delay_us * 1000),
              int(limit_us * 1000), res, None)
    return list(res)[:ctas]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("ctas", [2, 8, 16])
def test_sums_are_exact(ctas, form):
    assert _check(ctas, form, 1000) == [0] * ctas


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("ctas,who,at", [(2, 0, 0), (2, 1, 3), (8, 5, 2), (16, 15, 1)])
def test_a_cta_that_leaves_ends_the_others_waits(ctas, who, at, form):
    got = _check(ctas, form, 6, who, at, -1, 20_000)
    assert got == [TIMEOUT] * ctas
    assert _check(ctas, form, 10) == [0] * ctas
    assert float(torch.arange(1000, device="cuda", dtype=torch.float32).sum()) == 499500.0


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("ctas,who,at", [(2, 1, 0), (4, 0, 2), (8, 3, 5), (16, 7, 3)])
def test_a_cta_that_comes_late_learns_that_the_others_left(ctas, who, at, form):
    """The late CTA finds every total of the reduction it missed: it must not go on past the others' end,
    at a barrier in its loop, in its next reduction or (at = 5, the last) at its own end."""
    assert _check(ctas, form, 6, who, at, 30_000, 5_000) == [TIMEOUT] * ctas
    assert _check(ctas, form, 10) == [0] * ctas


@pytest.mark.parametrize("form", FORMS)
def test_threads_of_a_cta_agree_when_the_last_total_lands_as_time_runs_out(form):
    """The late CTA comes around the moment at which the others give up: whichever threads see the
    total first, a CTA goes on or gives up as one, and no sum that is used is wrong."""
    seen = set()
    for k in range(120):
        got = _check(4, form, 6, 1, 2, 200 + 2 * k, 300)
        assert got in ([0] * 4, [TIMEOUT] * 4), (k, got)
        seen.add(got[0])
    assert seen == {0, TIMEOUT}
