"""The shared slots of pinned host memory (csrc/mpm_pinned.h) with a fake
allocator, in a small host program: handles opened and closed one after the
other share one allocation, more handles than slots take further blocks that
are freed when they empty, a block never outlives its CUDA context (device
reset, its addresses handed out again, another device current at the close),
without context ids every block is freed, an allocation failure is passed on,
and threads may take and give at once.  And the engine makes no pinned
allocation of its own for a handle."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "edegpredict-engine-rotary_b200" / "csrc"

PROG = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>
#include "mpm_pinned.h"
using namespace mpmb;

struct World {
    uint64_t ctx = 1;
    bool known = true, fail = false;
    int allocs = 0, releases = 0;
    void* next = nullptr;   // the address the next allocation returns
    std::set<void*> live;
};
struct Ops {
    World* w;
    bool context(uint64_t* id) { *id = w->ctx; return w->known; }
    void* alloc(size_t n) {
        if (w->fail) return nullptr;
        void* p = w->next ? w->next : std::aligned_alloc(512, n);
        w->next = nullptr;
        ++w->allocs;
        w->live.insert(p);
        return p;
    }
    void release(void* p) {
        assert(w->live.erase(p) == 1);   // only what is allocated in the current world
        ++w->releases;
    }
};
using Slots = PinnedSlots<Ops>;

int main() {
    {   // one handle after another
        World w;
        Slots s(Ops{&w});
        for (int k = 0; k < 100; ++k) {
            void* p = s.take();
            assert(p && (uintptr_t)p % Slots::kSlotBytes == 0);
            s.give(p);
        }
        assert(w.allocs == 1 && w.releases == 0 && s.blocks() == 1);
    }
    {   // more handles than slots, closed in either order
        World w;
        Slots s(Ops{&w});
        for (int rev = 0; rev < 2; ++rev) {
            std::vector<void*> p;
            for (int k = 0; k < 3 * Slots::kSlots + 1; ++k) p.push_back(s.take());
            assert(std::set<void*>(p.begin(), p.end()).size() == p.size() && s.blocks() == 4);
            if (rev) p = std::vector<void*>(p.rbegin(), p.rend());
            for (void* q : p) s.give(q);
            assert(s.blocks() == 1 && (int)w.live.size() == 1);
        }
    }
    {   // a device reset: the block ends with its context, its address comes back
        World w;
        Slots s(Ops{&w});
        void* a = s.take();
        void* open_across = s.take();
        s.give(a);
        w.live.clear();
        w.ctx = 2;
        void* b = s.take();          // a new block, elsewhere
        assert(b != a && w.allocs == 2 && s.blocks() == 2);
        s.give(open_across);         // the old context's: nothing is freed
        assert(w.releases == 0);
        s.give(b);
        w.live.clear();
        w.ctx = 3;
        w.next = a;                  // the first block's address again
        void* c = s.take();
        assert(c == a && w.allocs == 3 && w.live.size() == 1);
        s.give(c);
        assert(s.take() == c && w.allocs == 3);
        s.give(c);
    }
    {   // two devices: each has its block; a close with the other one current frees nothing
        World w;
        Slots s(Ops{&w});
        void* a = s.take();
        w.ctx = 2;
        void* b = s.take();
        assert(w.allocs == 2);
        s.give(a);
        w.ctx = 1;
        s.give(b);
        assert(w.releases == 0 && s.take() == a && w.allocs == 2);
        w.ctx = 2;
        assert(s.take() == b && w.allocs == 2);
    }
    {   // no context ids: nothing is kept
        World w;
        w.known = false;
        Slots s(Ops{&w});
        void* a = s.take();
        void* b = s.take();
        assert(a != b && w.allocs == 2);
        s.give(a);
        s.give(b);
        assert(w.releases == 2 && s.blocks() == 0);
    }
    {   // out of memory
        World w;
        w.fail = true;
        Slots s(Ops{&w});
        assert(s.take() == nullptr && s.blocks() == 0);
    }
    {   // threads
        World w;
        Slots s(Ops{&w});
        std::vector<std::thread> t;
        for (int k = 0; k < 8; ++k)
            t.emplace_back([&] {
                for (int q = 0; q < 2000; ++q) {
                    void* p[9];
                    for (auto& x : p) { x = s.take(); *static_cast<void**>(x) = &x; }
                    for (auto& x : p) assert(*static_cast<void**>(x) == &x);
                    for (auto& x : p) s.give(x);
                }
            });
        for (auto& x : t) x.join();
        assert(s.blocks() <= 3 && w.live.size() == s.blocks());
    }
    std::puts("OK");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_slots(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROG)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(CSRC), str(src), "-o", str(exe), "-pthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stderr


def test_a_handle_allocates_no_pinned_memory_of_its_own():
    src = (CSRC / "mpm_engine.cu").read_text()
    engine = src[src.index("class Engine final"):]
    assert "pinned_take()" in engine and "cudaHostAlloc" not in engine and "cudaMallocHost" not in engine
