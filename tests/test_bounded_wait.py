"""The limit of the kernels' waits (csrc/bounded_wait.h), compiled for the CPU and
run against a clock and a completion flag that the test sets."""
import os
import subprocess

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <initializer_list>
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
    // A group's issuer: MMA k takes took[k] ticks from its issue; the barrier's
    // current phase is the number of completed ones.  Returns when the issuer may give
    // the accumulators back, and counts the waits that ran out.
    auto group = [](std::initializer_list<long long> took, int* ran_out) {
        long long now = 0, end = 0;
        int issued = 0;
        tvmc::GroupWaits w;
        auto poll = [&](uint32_t parity) {  // as mbarrier.test_wait: the phase of this parity is over
            const int complete = issued - (now < end);
            return (uint32_t)((complete & 1) ^ 1) == parity;
        };
        auto clock = [&] { return ++now; };
        *ran_out = 0;
        for (long long t : took) {
            if (!w.dead) {
                issued++;
                end = now + t;
            }
            *ran_out += !tvmc::group_wait(w, poll, clock, 100);
        }
        tvmc::group_drain(w, poll, clock, 100);
        return now >= end;
    };
    int ran_out;
    check(group({10, 20, 30}, &ran_out) && ran_out == 0, "three MMAs in time");
    check(group({10, 150, 5}, &ran_out) && ran_out == 1, "an odd MMA late: drained, nothing issued after it");
    check(group({150, 5}, &ran_out) && ran_out == 1, "an even MMA late: drained");
    check(!group({10, 100000}, &ran_out) && ran_out == 1, "an MMA that never ends: the drain is bounded too");
    return bad;
}
"""


def test_limit_and_last_poll(tmp_path):
    src, exe = tmp_path / "w.cpp", tmp_path / "w"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++20", "-O1", "-I", os.path.join(PKG, "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
