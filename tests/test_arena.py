"""Growth of a context's scratch against a device with little room (a host program against the
rules' header)."""
from __future__ import annotations

import subprocess

from thesiscode_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "mp_arena.h"
using namespace mpgpu;
struct Device {
    size_t size, used = 0;
    std::map<void*, size_t> blocks;
    int allocs = 0, fails = 0, frees = 0, asked = 0;
    char* next = (char*)4096;
    void* alloc(size_t bytes) {
        ++allocs;
        if (used + bytes > size) return ++fails, nullptr;
        void* p = next;
        next += bytes + 4096;
        used += bytes;
        blocks[p] = bytes;
        return p;
    }
    void free(void* p) {
        ++frees;
        used -= blocks.at(p);
        blocks.erase(p);
    }
    size_t room() { return ++asked, size - used; }
};
#define CHECK(x) if (!(x)) { std::printf("line %d: " #x "\n", __LINE__); return 1; }
// reserve_with's order of calls
static bool with(Arena& a, size_t base, size_t extra, Device& d, bool& ok) {
    const bool has = arena_try(a, base, base + extra, d);
    ok = has || arena_reserve(a, base, d);
    return has;
}
int main() {
    bool ok;
    {  // room for the need, not for the rest
        Device d{100};
        Arena a;
        CHECK(!with(a, 60, 50, d, ok) && ok && a.bytes == 60);
        void* p = a.p;
        const int allocs = d.allocs;
        for (int i = 0; i < 10; ++i) CHECK(!with(a, 60, 50, d, ok) && ok);
        CHECK(d.allocs == allocs && d.fails == 1 && d.frees == 0 && a.p == p);
        CHECK(!with(a, 60, 45, d, ok) && ok && a.p == p);  // a smaller one is tried once
        CHECK(!with(a, 60, 45, d, ok) && d.fails == 2 && d.frees == 0);
        d.size = 300;  // the device has room again
        CHECK(with(a, 60, 50, d, ok) && ok && a.bytes == 110 && d.used == 110 && d.blocks.size() == 1);
        CHECK(with(a, 60, 50, d, ok) && d.allocs == allocs + 2);
    }
    {  // a block that holds the need stays when the larger one is refused
        Device d{100};
        Arena a;
        CHECK(arena_reserve(a, 70, d));
        void* p = a.p;
        CHECK(!with(a, 60, 30, d, ok) && ok && a.p == p && d.frees == 0);
    }
    {  // one that does not hold it goes first, as ever
        Device d{100};
        Arena a;
        CHECK(arena_reserve(a, 40, d));
        CHECK(with(a, 60, 30, d, ok) && ok && a.bytes == 90 && d.used == 90);
        CHECK(!with(a, 95, 30, d, ok) && ok && a.bytes == 95);
        CHECK(!arena_reserve(a, 101, d) && !a.p && !a.bytes && d.used == 0);
        CHECK(arena_reserve(a, 10, d) && a.bytes == 10);
    }
    {  // room that no one block finds is not asked for in every call
        Device d{100};
        Arena a;
        CHECK(arena_reserve(a, 10, d));
        struct Split : Device {
            void* alloc(size_t bytes) { return ++allocs, bytes > 30 ? nullptr : Device::alloc(bytes); }
        } s;
        s.size = 100;
        Arena b;
        for (int i = 0; i < 5; ++i) CHECK(!arena_try(b, 20, 50, s));
        CHECK(s.allocs == 1);
    }
    return 0;
}
"""


def test_refused_sizes_are_not_asked_for_in_every_call(tmp_path):
    src, exe = tmp_path / "arena.cpp", tmp_path / "arena"
    src.write_text(PROGRAM)
    subprocess.run(["g++", *build.CXX_FLAGS, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
