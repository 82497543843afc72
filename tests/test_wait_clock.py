"""The clock of the clusters' bounded waits (csrc/wait_clock.cuh), compiled for the host: polls that keep
failing end the wait at its limit; a gap in which the kernel was set aside does not."""
import ctypes as ct
import shutil
import subprocess

import pytest

from warpcfd_gb300.build import CSRC

SRC = """
#include "wait_clock.cuh"
extern "C" int polls_until_over(const unsigned long long* now, int n, unsigned long long limit) {
    wcfd::WaitClock c(now[0]);
    for (int i = 1; i < n; ++i)
        if (c.over(now[i], limit)) return i;
    return 0;
}
"""
MS, S = 10**6, 10**9


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("clock")
    (d / "c.cpp").write_text(SRC)
    subprocess.run([gxx, "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "c.cpp"), "-o", str(d / "c.so")], check=True)
    return ct.CDLL(str(d / "c.so"))


def _over(lib, times, limit):
    a = (ct.c_uint64 * len(times))(*times)
    return lib.polls_until_over(a, len(times), ct.c_uint64(limit))


@pytest.mark.parametrize("step", [500, 10**5, MS])
def test_polls_that_keep_failing_end_the_wait(lib, step):
    limit = 20 * MS
    n = limit // step
    times = [7 * S + i * step for i in range(n + 10)]
    assert _over(lib, times, limit) == n + 1


def test_a_suspension_does_not(lib):
    limit = 1500 * MS
    before = [i * 2000 for i in range(100)]
    after = [before[-1] + 3600 * S + i * 2000 for i in range(100)]      # set aside for an hour
    assert _over(lib, before + after, limit) == 0
