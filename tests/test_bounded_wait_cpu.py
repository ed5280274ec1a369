"""The form of the kernels' bounded waits (csrc/bounded_wait.h), compiled for the host with a clock of its own.

What is waited for may arrive while the waiting thread is off the GPU for longer than the limit: the wait must
then see it, not report a time-out.  One that never comes is a time-out after the limit.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tomographic-image-reconstruction-algorithms_gb300", "csrc")

HARNESS = r"""
#include <cstdint>
#include <cstdio>
#include "bounded_wait.h"

// A row that arrives at time `at`; the n-th look at the clock jumps ahead by `jump`, each poll takes 1.
struct World {
    uint64_t now = 5, at = 0, jump = 0;
    int jump_at = -1, looks = 0, polls = 0;
    bool ready() { ++polls; ++now; return now > at; }
    uint64_t clock() { if (looks++ == jump_at) now += jump; return now; }
    bool wait(uint64_t limit) {
        return bounded_wait([&] { return ready(); }, [&] { return clock(); }, [&](uint64_t t0) { return clock() - t0 < limit; });
    }
};
static int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s\n", __LINE__, #c); ++fails; } } while (0)

int main() {
    { World w; CHECK(w.wait(100)); CHECK(w.polls == 1 && w.looks == 0); }              // there at once: no clock is read
    { World w; w.at = 40; CHECK(w.wait(100)); CHECK(w.polls < 100); }                  // within the limit
    { World w; w.at = UINT64_MAX; CHECK(!w.wait(100)); CHECK(w.polls <= 104); }        // never
    for (int n = 0; n < 20; ++n) {                                                     // off the GPU at the n-th look
        World w;
        w.at = 50; w.jump = 1000; w.jump_at = n;
        CHECK(w.wait(100));
    }
    { World w; w.at = UINT64_MAX; CHECK(!w.wait(0)); CHECK(w.polls == 2); }            // no time at all
    std::printf(fails ? "FAILED %d\n" : "OK\n", fails);
    return fails ? 1 : 0;
}
"""


def test_arrival_while_descheduled_is_not_a_timeout(tmp_path):
    src, exe = tmp_path / "wait_check.cpp", tmp_path / "wait_check"
    src.write_text(HARNESS)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-I" + CSRC, str(src), "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail("harness does not compile:\n" + r.stderr)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
