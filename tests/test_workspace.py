"""Growth of the library's cached workspaces and the numbers of its launches
(gmkbe_b200/csrc/workspace.h, compiled alone with g++), on the CPU: memory that
was allocated again counts as new, also where the allocator returns the same
address, and a buffer of numbered records is cleared before its first launch,
after growing, and when its numbers are used up."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include "workspace.h"
#include <cassert>
#include <cstdio>
#include <cstring>
// hands the same address out every time, with what was in it
static uint32_t store[64];
static int fail_next = 0, freed = 0;
static int alloc(void** p, size_t) {
    if (fail_next) { fail_next = 0; return -5; }
    *p = store;
    return 0;
}
static void release(void*) { ++freed; }

// a run over a buffer of records, as the library makes it; returns how many of
// its words would count as this launch's records before any is written
static uint32_t launch = 0;
static int stale(void** p, size_t* have, size_t need, uint32_t max) {
    bool fresh = false, clear = false;
    const int rc = gmk::grow_buffer(p, have, need, &fresh, alloc, release);
    if (fresh) launch = 0;
    if (rc) return rc;
    launch = gmk::next_launch(launch, max, &clear);
    if (clear) std::memset(*p, 0, *have);
    int n = 0;
    for (size_t i = 0; i < need / 4; ++i) n += static_cast<uint32_t*>(*p)[i] == launch;
    return n;
}

int main() {
    void* p = nullptr;
    size_t have = 0;
    for (uint32_t i = 0; i < 64; ++i) store[i] = i % 5;      // what others left there
    assert(stale(&p, &have, 32, 0xFFFFFFFFu) == 0 && launch == 1 && have == 32);
    for (uint32_t i = 0; i < 8; ++i) store[i] = launch;       // this launch's records
    assert(stale(&p, &have, 32, 0xFFFFFFFFu) == 0 && launch == 2);
    assert(stale(&p, &have, 16, 0xFFFFFFFFu) == 0 && launch == 3 && have == 32 && freed == 0);
    // larger, at the same address: cleared, whatever the new part holds
    for (uint32_t i = 8; i < 64; ++i) store[i] = 1 + i % 4;
    assert(stale(&p, &have, 256, 0xFFFFFFFFu) == 0 && launch == 1 && have == 256 && freed == 1);
    // numbers used up
    for (uint32_t i = 0; i < 64; ++i) store[i] = 1 + i % 8;
    launch = 8;
    assert(stale(&p, &have, 256, 9) == 0 && launch == 9);
    assert(stale(&p, &have, 256, 9) == 0 && launch == 1);
    // a failed growth leaves nothing behind, and what follows starts cleared
    store[0] = 1;
    fail_next = 1;
    assert(stale(&p, &have, 512, 9) == -5 && p == nullptr && have == 0 && launch == 0);
    assert(stale(&p, &have, 128, 9) == 0 && launch == 1 && store[0] == 0);
    std::puts("ok");
    return 0;
}
"""


def test_grown_memory_counts_as_new_and_is_cleared(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    src = tmp_path / "drv.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "drv"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "gmkbe_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr
