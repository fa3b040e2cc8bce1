"""The ring of shared states of the small graphs' search
(gmkbe_b200/csrc/state_ring.h, compiled alone with g++), on the CPU: warps that
take tickets, hand work on, wait for slots and read them, one memory access at a
time in random order, some of them held up for long.  Every record is read once,
none is written over before it was read, the work never stalls, and tickets go
round the ring many times; the marks go on from launch to launch."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include "state_ring.h"
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
using namespace gmk;
typedef unsigned long long u64;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)

struct Slot { uint32_t mark; u64 ticket; int work; bool unread; };
enum Step { IDLE, WAIT, READ, BUSY, SEE, NOW, AGAIN, RESERVE, SPIN, WRITE, MARK };
struct Warp { Step step = IDLE; u64 ticket = 0, seen = 0, at = 0; int work = 0, n = 0, i = 0, want = 0, hold = 0; };

// One launch of `warps` warps over `total` units of work, all with warp 0 at first.
static u64 launch(std::vector<Slot>& slots, const StateRing& ring, int warps, long total, unsigned seed) {
    std::mt19937 rng(seed);
    auto pick = [&](int n) { return (int)(rng() % n); };
    std::vector<Warp> w(warps);
    w[0].step = BUSY;
    w[0].work = (int)total;
    u64 tail = 0, claim = 0;
    long done = 0, steps = 0;
    while (done < total) {
        CHECK(++steps < 4000 * total + 1000000);
        Warp& x = w[pick(warps)];
        if (x.hold > 0) { --x.hold; continue; }
        if (pick(400) == 0) { x.hold = pick(3000); continue; }
        Slot& mine = slots[ring.slot(x.ticket)];
        switch (x.step) {
            case IDLE: x.ticket = claim++; x.step = WAIT; break;
            case WAIT: if (mine.mark == ring.ready(x.ticket)) x.step = READ; break;
            case READ:
                CHECK(mine.ticket == x.ticket && mine.unread);
                x.work = mine.work;
                mine.unread = false;
                mine.mark = ring.ready(x.ticket) + 1;
                x.step = BUSY;
                break;
            case BUSY:
                if (x.work == 0) { x.step = IDLE; break; }
                // (before: the reserved tickets, then the claimed ones)
                if (x.work > 1 && pick(2)) { x.seen = tail; x.step = SEE; break; }
                --x.work;
                ++done;
                break;
            case SEE:
                x.want = claim > x.seen ? (int)(claim - x.seen < 32 ? claim - x.seen : 32) : 0;
                x.step = x.want == 0 ? BUSY : ring.early(x.seen) ? RESERVE : NOW;
                break;
            case NOW: x.seen = claim; x.step = AGAIN; break;
            case AGAIN:
                x.want = x.seen > tail ? (int)(x.seen - tail < 32 ? x.seen - tail : 32) : 0;
                x.step = x.want == 0 ? BUSY : RESERVE;
                break;
            case RESERVE:
                x.n = x.want < (int)kRingShare ? x.want : (int)kRingShare;
                if (x.n > x.work - 1) x.n = x.work - 1;
                if (x.n <= 0) { x.step = BUSY; break; }
                x.at = tail;
                tail += x.n;
                CHECK(tail <= ring.slots() || tail <= claim + (u64)kRingShare * warps);
                x.i = 0;
                x.step = SPIN;
                break;
            case SPIN: {
                const u64 t = x.at + x.i;
                if (ring.first(t) || ring.free(t, slots[ring.slot(t)].mark)) x.step = WRITE;
                break;
            }
            case WRITE: {
                Slot& s = slots[ring.slot(x.at + x.i)];
                CHECK(!s.unread);
                s.ticket = x.at + x.i;
                s.work = 1 + (x.work > 40 && pick(40) == 0 ? pick(x.work / 4) : 0);
                if (s.work > x.work - (x.n - x.i)) s.work = 1;
                x.work -= s.work;
                x.step = MARK;
                break;
            }
            case MARK: {
                Slot& s = slots[ring.slot(x.at + x.i)];
                s.unread = true;
                s.mark = ring.ready(x.at + x.i);
                x.step = ++x.i < x.n ? SPIN : BUSY;
                break;
            }
        }
    }
    for (Slot& s : slots) CHECK(!s.unread);
    return tail;
}

int main() {
    bool clear;
    // sizes: enough slots for the warps, marks from the last launch's on
    for (uint64_t n : {1, 31, 32, 33, 4736, 5000}) {
        const StateRing r = ring_begin(n, 0, &clear);
        CHECK(clear && r.base == 1 && r.slots() >= kRingWarp * n);
        CHECK(r.slots() < 2 * kRingWarp * n);
        const StateRing s = ring_begin(n, 77, &clear);
        CHECK(!clear && s.base == 77 && s.shift == r.shift);
        CHECK(!r.free(r.slots(), 0) && !r.free(r.slots(), r.ready(0)) && r.free(r.slots(), r.ready(0) + 1));
    }
    CHECK(ring_next(StateRing{5, 8}, 0) == 5 && ring_next(StateRing{5, 8}, 1) == 7);
    CHECK(ring_next(StateRing{5, 8}, 256) == 7 && ring_next(StateRing{5, 8}, 257) == 9);
    CHECK(ring_next(StateRing{(1u << 31) - 2, 8}, 1) == 0);

    // launches one after the other over the same slots, with rings of two sizes:
    // 64 slots a warp, the fewest that early() goes with
    for (unsigned seed = 0; seed < 12; ++seed) {
        std::vector<Slot> slots(1024, Slot{0, 0, 0, false});
        uint32_t base = 0;
        u64 rounds = 0;
        for (int l = 0; l < 6; ++l) {
            const int warps = l % 3 == 0 ? 16 : l % 3 == 1 ? 4 : 2;
            StateRing ring = ring_begin(warps, base, &clear);
            ring.shift = warps == 16 ? 10 : warps == 4 ? 8 : 7;
            if (clear) for (Slot& s : slots) s.mark = 0;
            const u64 tail = launch(slots, ring, warps, 150000, 100 * seed + l);
            rounds += tail >> ring.shift;
            base = ring_next(ring, tail);
            for (const Slot& s : slots) CHECK(s.mark < base);
        }
        CHECK(rounds > 20);
    }
    std::puts("ok");
    return 0;
}
"""


def test_shared_states_go_round_the_ring(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    src = tmp_path / "drv.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "drv"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "gmkbe_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
