"""The place of an item in a warp's pool of paths (csrc/pool_index.h), compiled for the host.

A time-limited render's pool holds all strata of a tile.  From 178,956,987 items on (6.39 M strata of a
7x4 tile) the high multiply that replaces the division by 28 is one too large, so the rule has to divide
there: the quotient is checked against the plain division at the ends of every pool's range and around
the place where the multiply stops serving it.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "luminara_b200", "csrc")

MAIN = """
#include <cstdio>
#include <cstdlib>
#include "pool_index.h"
int main(int, char** v) {
    const uint32_t n = strtoul(v[1], 0, 10);
    const uint64_t items = strtoull(v[2], 0, 10);
    const uint32_t magic = lum::pool_magic(n, items);
    uint64_t bad = 0, last = items - 1;
    auto at = [&](uint64_t i) { if (i <= last && lum::pool_stratum((uint32_t)i, n, magic) != i / n) ++bad; };
    for (uint64_t k = 0; k < 4096; ++k) { at(k); at(last - (k < last ? k : last)); }
    for (uint64_t q = 1; q <= last / n; q += 1 + last / n / 50000) { at(q * n - 1); at(q * n); }   // edges of strata
    for (uint64_t i = 178956970; i < 178957100; ++i) at(i);
    printf("%llu %u\\n", (unsigned long long)bad, magic);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-o", str(d / "main"), str(d / "main.cpp")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("strata", [1, 16, 9216, 6_391_321, 6_391_322, 12_000_000, 17_000_000, 2 ** 27 - 1])
def test_quotient_is_the_division(program, strata):
    for n in range(1, 33):
        items = min(n * strata, 2 ** 32 - 1)
        bad, magic = map(int, subprocess.run([program, str(n), str(items)], check=True, capture_output=True,
                                             text=True).stdout.split())
        assert bad == 0, (n, items, magic)
        # the multiply where it serves the whole pool, the division elsewhere
        assert (magic != 0) == (n > 1 and items * n <= 2 ** 32)


def test_the_multiply_alone_would_be_wrong():
    magic = (2 ** 32 - 1) // 28 + 1
    assert (178956987 * magic) >> 32 == 178956987 // 28 + 1
