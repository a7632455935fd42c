"""The rules of the library's block cache (csrc/block_cache.h), with a counting
allocator in place of the device's."""
import os
import subprocess

from conftest import ROOT

SRC = r"""
#include "block_cache.h"
#include <cassert>
#include <cstdio>
#include <cstdint>
#include <map>

static std::map<void*, size_t> live;
static size_t room = (size_t)1 << 40;
static int allocs = 0;
static size_t used() { size_t n = 0; for (auto& e : live) n += e.second; return n; }
static int get(void** p, size_t n) {
    if (used() + n > room) return 2;
    *p = (void*)(uintptr_t)++allocs;   // (addresses are never used twice)
    live[*p] = n;
    return 0;
}
static void release(void* p) { assert(live.erase(p) == 1); }
static const size_t MB = 1 << 20;

int main() {
    void *p, *q;
    size_t n, m;
    {   // a block goes to a request of its size, on its device
        rms::BlockCache c(get, release, 100 * MB);
        assert(c.take(10 * MB, 0, &p, &n) == 0 && n == 10 * MB);
        c.give(p, n, 0);
        assert(c.held(0) == 10 * MB && c.held(1) == 0);
        assert(c.take(10 * MB, 1, &q, &m) == 0 && q != p);
        c.give(q, m, 1);
        assert(c.take(9 * MB, 0, &q, &m) == 0 && q == p && m == 10 * MB && c.held(0) == 0);
        c.give(q, m, 0);
        assert(c.take(7 * MB, 0, &q, &m) == 0 && q != p);   // over a quarter and 1 MB larger
        c.give(q, m, 0);
        // all of it back
        assert(c.trim() == 27 * MB && live.empty() && c.held(0) == 0 && c.trim() == 0);
    }
    {   // bounded: the oldest go first, and a block larger than the bound is not kept
        rms::BlockCache c(get, release, 25 * MB);
        void* b[3];
        for (auto& x : b) assert(c.take(10 * MB, 0, &x, &n) == 0);
        for (auto& x : b) c.give(x, n, 0);
        assert(c.held(0) == 20 * MB && !live.count(b[0]) && live.count(b[1]) && live.count(b[2]));
        assert(c.take(30 * MB, 0, &p, &n) == 0);
        c.give(p, n, 0);
        assert(!live.count(p));
        c.trim();
    }
    {   // a block 256 requests have passed over goes, whether or not anything is given back
        rms::BlockCache c(get, release, 100 * MB);
        assert(c.take(50 * MB, 0, &p, &n) == 0);
        c.give(p, n, 0);
        void* small[257];
        for (int k = 0; k < 257; ++k) {
            assert(live.count(p));
            assert(c.take(64, 0, &small[k], &m) == 0);
        }
        assert(!live.count(p) && c.held(0) == 0);
        for (void* x : small) c.give(x, 64, 0);
        c.trim();
    }
    {   // the block asked for is not dropped on the way
        rms::BlockCache c(get, release, 100 * MB);
        assert(c.take(50 * MB, 0, &p, &n) == 0);
        c.give(p, n, 0);
        void* small[256];
        for (void*& x : small) assert(c.take(64, 0, &x, &m) == 0);
        assert(c.take(50 * MB, 0, &q, &m) == 0 && q == p && live.count(p));
        c.give(q, m, 0);
        for (void* x : small) c.give(x, 64, 0);
        c.trim();
    }
    {   // an allocation that fails empties the cache and is tried again
        rms::BlockCache c(get, release, 100 * MB);
        room = 60 * MB;
        assert(c.take(50 * MB, 0, &p, &n) == 0);
        c.give(p, n, 0);
        assert(c.take(20 * MB, 0, &q, &m) == 0 && !live.count(p));
        const int before = allocs;
        assert(c.take(50 * MB, 0, &p, &n) == 2 && p == nullptr && allocs == before);
        c.give(q, m, 0);
        c.trim();
    }
    assert(live.empty());
    std::puts("ok");
}
"""


def test_rules(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    csrc = os.path.join(ROOT, "monte-carlo-simulation-3d-rms_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", csrc, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stderr


def test_trim_leaves_nothing():
    from rms_b200 import engine
    engine.trim_memory()
    assert engine.trim_memory() == (0, 0)
