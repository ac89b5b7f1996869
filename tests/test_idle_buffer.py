"""Device memory kept between calls (csrc/idle_buffer.h), compiled for the host over an allocator with a
limit: the buffer goes back when an allocation finds no memory, before a larger one replaces it, and
with the last owner; every allocation of device memory goes through the helper that retries."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "luminara_b200", "csrc")

MAIN = """
#include <cassert>
#include <cstdio>
#include <map>
#include "idle_buffer.h"
static std::map<void*, size_t> live;
static size_t held = 0, peak = 0, limit = 100, next_id = 1;
static void* get(size_t n) {
    if (held + n > limit) return nullptr;
    void* p = (void*)(next_id++ * 16);
    live[p] = n;
    held += n;
    if (held > peak) peak = held;
    return p;
}
static void release(void* p) {
    assert(live.count(p));
    held -= live[p];
    live.erase(p);
}
using lum::IdleBuffer;
// what a call does: the idle buffer, or a new one with one more try
static void* call(IdleBuffer& b, size_t* n) {
    if (void* p = b.take(n)) return p;
    void* p = nullptr;
    const int e = lum::alloc_or_release(2, [&] { return (p = get(*n)) ? 0 : 2; }, [&] { b.give_back(); });
    return e == 0 ? p : nullptr;
}
int main() {
    IdleBuffer b(release, 80);
    b.add_owner();
    size_t n = 60;
    void* p = call(b, &n);
    b.put(p, n);
    assert(held == 60);
    n = 50;
    assert(call(b, &n) == p && n == 60);                  // reused, with its own size
    b.put(p, n);
    {   // another allocation that would not fit beside the idle buffer
        void* q = nullptr;
        int tries = 0;
        auto alloc = [&] { ++tries; return (q = get(70)) ? 0 : 2; };
        assert(lum::alloc_or_release(2, alloc, [&] { b.give_back(); }) == 0 && tries == 2 && held == 70);
        release(q);
        tries = 0;
        limit = 10;
        assert(lum::alloc_or_release(2, alloc, [&] { b.give_back(); }) == 2 && tries == 2);   // there is none
        tries = 0;
        assert(lum::alloc_or_release(2, [&] { ++tries; return 7; }, [&] { assert(false); }) == 7 && tries == 1);
        limit = 100;
    }
    n = 40;
    p = call(b, &n);
    b.put(p, n);
    peak = held;
    n = 70;
    p = call(b, &n);                                      // the smaller one is not held beside it
    assert(p && peak == 70 && held == 70);
    size_t m = 20;
    void* q = call(b, &m);                                // a second call at the same time
    assert(q && q != p && m == 20);
    b.put(p, n);
    b.put(q, m);                                          // the larger one stays
    assert(held == 70);
    b.give_back();
    n = 90;
    p = call(b, &n);
    b.put(p, n);                                          // above what is kept
    assert(held == 0);
    n = 30;
    b.add_owner();
    p = call(b, &n);
    b.put(p, n);
    b.remove_owner();
    assert(held == 30);
    b.remove_owner();                                     // the last owner
    assert(held == 0 && live.empty());
    puts("ok");
}
"""


def test_what_is_kept_goes_back(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "main"),
                    str(tmp_path / "main.cpp")], check=True)
    r = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stderr


def test_every_device_allocation_retries():
    calls = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".cpp", ".h")):
            with open(os.path.join(CSRC, name)) as f:
                code = re.sub(r"//.*", "", f.read())
            calls += [(name, c) for c in re.findall(r"\b(cudaMalloc|cudaMallocFromPoolAsync|cudaMallocAsync)\(", code)]
    # one place each, inside alloc_or_release
    assert calls == [("host.cpp", "cudaMallocFromPoolAsync"), ("host.cpp", "cudaMalloc")]
