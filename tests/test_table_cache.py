"""Which tone-map byte tables are built and kept (csrc/table_cache.h), compiled for the host: a pair without
a table is tried once, takes no slot, and neither it nor a swept gamma of chains with optional steps
keeps a new pair of the common chain from its table."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "luminara_b200", "csrc")

MAIN = """
#include <cassert>
#include <cstdio>
#include "table_cache.h"
using Cache = lum::TableCache<int>;
static int tries = 0;
// one call with the pair (0, gamma), whose table exists or not: its table, 0 for none
static int call(Cache& c, long long gamma, bool graded, bool fits, int device = 0) {
    bool known = false;
    if (const int* t = c.find(device, 0, gamma, &known)) return *t;
    const int slot = c.free_slot(device, graded);
    if (known || slot < 0) return 0;
    ++tries;
    if (!fits) { c.add_failed(device, 0, gamma); return 0; }
    c.add(device, 0, gamma, slot, (int)gamma);
    return (int)gamma;
}
int main() {
    {
        Cache c;
        for (int k = 0; k < 40; ++k) assert(call(c, 4, k & 1, false) == 0);
        assert(tries == 1);                                       // remembered
        for (int k = 0; k < 16; ++k) assert(call(c, 100 + k, false, true) == 100 + k);
        assert(call(c, 200, false, true) == 0);                   // no slot left, whatever failed before
        assert(call(c, 200, false, true, 1) == 200);              // another device
        for (int k = 0; k < 16; ++k) assert(call(c, 100 + k, true, true) == 100 + k);
        tries = 0;
        for (int k = 0; k < 1000; ++k) call(c, 1000 + k, true, true);
        assert(tries == Cache::kGraded);
    }
    {
        Cache c;
        tries = 0;
        for (int k = 0; k < 1000; ++k) assert((call(c, 1000 + k, true, true) != 0) == (k < Cache::kGraded));
        for (int k = 0; k < 16; ++k) assert(call(c, 100 + k, false, true) == 100 + k);   // all of the common chain's
        bool known = false;
        for (long long g = 1000; g < 1000 + Cache::kGraded; ++g) assert(*c.find(0, 0, g, &known) == g);
    }
    {
        Cache c;
        tries = 0;
        for (int k = 0; k < 1000; ++k) call(c, 1000 + k, true, false);
        assert(tries == (int)Cache::kMaxFailed);
        for (int r = 0; r < 3; ++r)
            for (int k = 0; k < 8; ++k) assert(call(c, 5000 + k, false, false) == 0);
        assert(tries == (int)Cache::kMaxFailed + 8);
        assert(call(c, 7, false, true) == 7);
    }
    puts("ok");
}
"""


def test_tables_and_failures(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "main"),
                    str(tmp_path / "main.cpp")], check=True)
    r = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stderr
