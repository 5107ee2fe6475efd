"""The pool of page-locked result slots (scp_b200/csrc/result_slots.h) on the
CPU, over a counting allocator: no slot is handed out twice, blocks that are no
longer held are given back, other contexts' blocks are left alone."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scp_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>
#include <vector>
#include "result_slots.h"

static int live = 0, calls = 0;
static bool refuse = false;
struct Mem {
    static double *alloc(size_t n) { if (refuse) return nullptr; live++; calls++; return (double *)std::malloc(n); }
    static void free(double *p) { live--; std::free(p); }
};
#define REQUIRE(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    using Pool = scp::SlotPool<Mem, 96>;
    constexpr int B = scp::SlotBlock::kSlots;
    {
        Pool p;
        std::vector<scp::ResultSlot *> held;
        std::set<double *> where;
        for (int i = 0; i < 5 * B + 1; i++) {
            held.push_back(p.take(1));
            REQUIRE(where.insert(held.back()->p).second);
        }
        REQUIRE(live == 6);
        for (auto *r : held) p.give(r, 1);
        REQUIRE(live == 1);                      // the last empty block is kept for the next handle
        for (int i = 0; i < 1000; i++) p.give(p.take(1), 1);
        REQUIRE(live == 1 && calls == 6);        // and no pinning per handle
    }
    live = calls = 0;
    {   // a block of a context that is gone: its slots come back, its memory is not touched
        Pool p;
        scp::ResultSlot *old = p.take(7), *now = p.take(8);
        REQUIRE(live == 2 && old->p != now->p);
        p.give(old, 8);
        REQUIRE(live == 2);
        scp::ResultSlot *more = p.take(8);
        REQUIRE(more->block == now->block);
        refuse = true;
        REQUIRE(p.take(9) == nullptr);
        refuse = false;
        REQUIRE(p.take(9) != nullptr);
    }
    {   // from several threads
        Pool p;
        std::vector<std::thread> t;
        for (int k = 0; k < 8; k++)
            t.emplace_back([&p] {
                for (int i = 0; i < 200; i++) {
                    std::vector<scp::ResultSlot *> h;
                    for (int q = 0; q < 100; q++) { h.push_back(p.take(1)); h.back()->p[0] = q; }
                    for (auto *r : h) p.give(r, 1);
                }
            });
        for (auto &x : t) x.join();
    }
    std::puts("ok");
}
"""


def test_slot_pool(tmp_path):
    src, exe = tmp_path / "slots.cc", tmp_path / "slots"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.stdout.strip() == "ok", r.stdout + r.stderr
