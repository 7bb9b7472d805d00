"""The bound of the persistent kernels' waits (csrc/wait_clock.h, host build): it
runs out after the time that the waiting thread itself polled, and not because
another program had the GPU for a while."""
from __future__ import annotations

import ctypes as C
import subprocess

import pytest

from conftest import ROOT

SRC = """
#include "wait_clock.h"
extern "C" int64_t polls_until_over(uint64_t step, uint64_t every, uint64_t gap, uint64_t limit, uint64_t most) {
    uint64_t now = 1000;
    pc::WaitClock clock(now);
    for (uint64_t i = 1; i <= most; ++i) {
        now += step + (every && i % every == 0 ? gap : 0);
        if (clock.over(now, limit)) return (int64_t)i;
    }
    return -1;
}
"""


@pytest.fixture(scope="module")
def polls(tmp_path_factory):
    d = tmp_path_factory.mktemp("wait_clock")
    (d / "w.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "partitionandconquer_b200" / "csrc"),
                    str(d / "w.cpp"), "-o", str(d / "w.so")], check=True)
    fn = C.CDLL(str(d / "w.so")).polls_until_over
    fn.argtypes, fn.restype = [C.c_uint64] * 5, C.c_int64
    return fn


def test_steady_polls_run_out_at_the_limit(polls):
    assert polls(1000, 0, 0, 4_000_000_000, 10_000_000) == 4_000_001


def test_gaps_hardly_count(polls):
    # one gap of 10 s, and a thousand of 2 ms: neither is 4 s of polling
    assert polls(1000, 500, 10_000_000_000, 4_000_000_000, 999) == -1
    assert polls(1000, 10, 2_000_000, 4_000_000_000, 10_000) == -1


def test_still_bounded_with_gaps_only(polls):
    assert polls(0, 1, 5_000_000, 4_000_000_000, 100_000) == 40_001
