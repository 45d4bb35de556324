"""The kernels' limit on a wait counts the time spent polling, and not the time
that the process was off the GPU between two polls (the header, compiled for the
host)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "meshode_gb300", "csrc")
CODE = r"""
#include "mo_wait.cuh"
// the number of the first of n clock readings at which the wait is over, or -1
extern "C" int first_over(const unsigned long long* t, int n) {
    mo::WaitLimit limit((unsigned)t[0]);
    for (int k = 1; k < n; ++k)
        if (limit.over((unsigned)t[k])) return k;
    return -1;
}
"""


@pytest.fixture(scope="module")
def first_over(tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    src, so = str(d / "w.cc"), str(d / "w.so")
    with open(src, "w") as f:
        f.write(CODE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, src, "-o", so], check=True)
    fn = ctypes.CDLL(so).first_over

    def call(times):
        return fn((ctypes.c_ulonglong * len(times))(*times), len(times))

    return call


@pytest.mark.parametrize("start", [0, 1 << 32, (1 << 32) - 1000, 123 << 40])
@pytest.mark.parametrize("poll", [500_000, 1_000_000, 7_000_003])
def test_two_seconds_of_polling(first_over, start, poll):
    k = first_over([start + i * poll for i in range(2_000_000_000 // poll + 3)])
    assert (k - 1) * poll <= 2_000_000_000 < k * poll


@pytest.mark.parametrize("away", [3_000_000_000, 10_000_000_000, 3600 * 10 ** 9])
def test_time_away_does_not_count(first_over, away):
    poll = 1_000_000
    times = [i * poll for i in range(100)]
    times += [times[-1] + away + i * poll for i in range(1000)]
    assert first_over(times) == -1
    times += [times[-1] + i * poll for i in range(1000)]
    assert first_over(times) > 0  # it still ends
