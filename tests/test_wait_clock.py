"""The clock of the waits inside kernels (csrc/wait_clock.h), compiled for the
host: a wait that polls gives up at its limit, time spent switched out does not
count, and the low word's wrap changes nothing."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIMIT = 1 << 31
STEP = 1 << 20  # what a gap between two looks counts at most

SRC = """
#include "wait_clock.h"
// The look (from 1 on) at which a wait gives up, 0 if none of the n does.
extern "C" int first_pass(const unsigned long long* at, int n, unsigned limit) {
  WaitClock w;
  for (int i = 0; i < n; i++)
    if (w.passed((uint32_t)at[i], limit)) return i + 1;
  return 0;
}
"""


@pytest.fixture(scope="module")
def first_pass(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no host compiler"
    d = tmp_path_factory.mktemp("wait_clock")
    (d / "w.cpp").write_text(SRC)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "flock_challenge_gb300", "csrc"),
                    str(d / "w.cpp"), "-o", str(d / "w.so")], check=True)
    f = ctypes.CDLL(str(d / "w.so")).first_pass

    def run(at, limit):
        return f((ctypes.c_ulonglong * len(at))(*at), len(at), ctypes.c_uint(limit))
    return run


def test_a_polling_wait_gives_up_at_its_limit(first_pass):
    for start in (0, (1 << 32) - 5000, 123456789012345):  # the low word wraps in all three
        looks = [start + i * (STEP // 4) for i in range(LIMIT // (STEP // 4) + 10)]
        assert first_pass(looks, LIMIT) == LIMIT // (STEP // 4) + 2  # the first look past the limit
    assert first_pass([7, 8, 9, 10], 1) == 3
    assert first_pass([7, 1007], 300) == 2


def test_time_switched_out_does_not_count(first_pass):
    gap = 4 * 10**9 + 77  # two seconds away, more than the limit
    assert first_pass([0, gap, gap + 1000], LIMIT) == 0
    assert first_pass([0, (1 << 32) - 1], LIMIT) == 0
    # a thousand time slices away, a little polling between
    at, t = [], 0
    for _ in range(1000):
        t += 4 * 10**6
        at += [t + 500 * k for k in range(4)]
        t += 2000
    assert first_pass(at, LIMIT) == 0


def test_the_longest_wait_does_not_overflow(first_pass):
    assert first_pass([i * (STEP + 9) for i in range(3000)], LIMIT) == LIMIT // STEP + 2
