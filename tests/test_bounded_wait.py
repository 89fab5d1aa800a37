"""The limit of the kernels' waits (csrc/bounded_wait.h), compiled for the CPU and
run against a clock and a completion flag that the test sets."""
import os
import subprocess

from conftest import PKG

SRC = r"""
#include <cstdio>
#include "bounded_wait.h"
// args of run: the clock's step per reading, the reading at which one long hold-up
// of `hold` ticks begins, and the time at which the awaited work completes
static bool run(long long step, int held_at, long long hold, long long done_at, long long limit, int* polls) {
    long long now = 0;
    int readings = 0;
    *polls = 0;
    return tvmc::bounded_wait([&] { ++*polls; return now >= done_at; },
                              [&] { if (++readings == held_at) now += hold; return now += step; }, limit);
}
int main() {
    int polls, bad = 0;
    auto check = [&](bool ok, const char* what) { if (!ok) { std::printf("%s\n", what); bad++; } };
    check(run(1, 0, 0, 0, 100, &polls) && polls == 1, "complete at the first poll");
    check(run(1, 0, 0, 50, 100, &polls), "completes within the limit");
    check(!run(1, 0, 0, 1000, 100, &polls) && polls < 110, "never completes: gives up at the limit");
    check(run(1, 2, 1000, 500, 100, &polls), "held up past the limit while the work completed");
    check(!run(1, 2, 1000, 5000, 100, &polls), "held up past the limit, work not complete");
    check(!run(1, 0, 0, 1000, 0, &polls) && polls == 2, "no limit at all: two polls");
    return bad;
}
"""


def test_limit_and_last_poll(tmp_path):
    src, exe = tmp_path / "w.cpp", tmp_path / "w"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++20", "-O1", "-I", os.path.join(PKG, "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
