"""Which host transfers take the pinned staging buffers (csrc/staging_rule.h), compiled for the host."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "luminara_b200", "csrc")

MAIN = """
#include <cassert>
#include <cstdio>
#include <initializer_list>
#include "staging_rule.h"
using lum::StagingRule;
using U = lum::StagingUse;
constexpr size_t MB = 1u << 20;
constexpr int64_t ms = 1000000;
static int64_t clock_ns = 0;
// a call of 0.3 ms, `gap` after the one before it
static bool call(StagingRule& r, U use, size_t bytes, bool ready, int64_t gap) {
    clock_ns += gap;
    const bool staged = r.begin(use, bytes, ready, clock_ns);
    clock_ns += 3 * ms / 10;
    r.end(bytes, clock_ns);
    return staged;
}
int main() {
    for (U u : {U::Frame, U::Rays}) {   // a call by itself: from 8 MB on
        StagingRule r;
        assert(!call(r, u, 8 * MB - 1, true, 100 * ms) && call(r, u, 8 * MB, true, 100 * ms));
        // in a row: from 1 MB on, after the first calls of each row
        for (int row = 0; row < 3; ++row)
            for (int k = 0; k < 20; ++k) {
                const bool staged = call(r, u, 2 * MB, true, k ? ms : 50 * ms);
                assert(staged == (k >= StagingRule::kRow));
            }
        for (int k = 0; k < 100; ++k) assert(!call(r, u, MB - 1, true, 0));
        // pairs of calls, and calls of 3 ms apart, never make a row
        for (int k = 0; k < 100; ++k) assert(!call(r, u, 2 * MB, true, k & 1 ? ms : 10 * ms));
        for (int k = 0; k < 100; ++k) assert(!call(r, u, 2 * MB, true, 3 * ms));
        // short calls in between neither make nor break one
        for (int k = 0; k < 20; ++k) {
            assert(!call(r, u, 1000, true, 0));
            assert(call(r, u, 2 * MB, true, k ? 0 : 50 * ms) == (k >= StagingRule::kRow));
        }
    }
    {   // the planes of AOVs
        StagingRule r;
        assert(!call(r, U::Planes, 3 * MB - 1, true, 100 * ms) && call(r, U::Planes, 3 * MB, true, 100 * ms));
    }
    {   // a process's first calls do not wait for the buffers' allocation, but for frames of 8 MB
        StagingRule r;
        assert(!call(r, U::Rays, 48 * MB, false, ms) && !call(r, U::Rays, 16 * MB, false, ms));
        assert(call(r, U::Rays, 8 * MB, false, ms));
        StagingRule f;
        for (int k = 0; k < 12; ++k) assert(!call(f, U::Frame, 5 * MB, false, ms));
        assert(call(f, U::Frame, 8 * MB, false, 100 * ms));
        StagingRule g;
        int direct = 0;
        while (!call(g, U::Rays, 5 * MB, false, 0)) ++direct;
        assert(direct == StagingRule::kRow + 12);
    }
    puts("ok");
}
"""


def test_rule(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "main"),
                    str(tmp_path / "main.cpp")], check=True)
    r = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stderr
