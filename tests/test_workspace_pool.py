"""Workspaces kept between calls: what the pool frees and what it only
forgets.  The pool itself runs on the CPU against a stand-in for CUDA's
contexts; on the GPU a program resets its context between two calls."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "necsim-rust_b200", "csrc")

PROGRAM = r"""
#include "workspace_pool.h"

#include <cstdio>
#include <map>
#include <vector>

static std::map<int, unsigned long long> context_of;  // device -> its context now
static std::vector<int> freed, dropped;

struct Contexts {
    static unsigned long long of(int device) { return context_of[device]; }
};
struct Space {
    int id, device;
    unsigned long long context = 0;
    size_t size;
    Space(int i, int d, size_t s) : id(i), device(d), size(s) {}
    ~Space() { freed.push_back(id); }
    size_t bytes() const { return size; }
    void drop_host_memory() { dropped.push_back(id); }
};
using Pool = necsim::WorkspacePool<Space, Contexts>;

static void show(const char *what) {
    std::printf("%s freed", what);
    for (int i : freed) std::printf(" %d", i);
    std::printf(" forgotten");
    for (int i : dropped) std::printf(" %d", i);
    std::printf("\n");
    freed.clear();
    dropped.clear();
}
static std::unique_ptr<Space> space(int i, int d, size_t s = 10) { return std::unique_ptr<Space>(new Space(i, d, s)); }
static int take(Pool &p, int device) {
    auto w = p.take(device, [](const Space &s) -> unsigned long long { return s.size; });
    const int id = w ? w->id : -1;
    (void)w.release();
    return id;
}

int main() {
    context_of = {{0, 7}, {1, 9}};
    {
        Pool p;
        p.put(space(1, 0), 100);
        p.put(space(2, 1), 100);
        context_of[0] = 8;  // device 0 was reset
        std::printf("%d ", (int)p.empty_out());
        show("emptied after a reset:");
        std::printf("%d ", (int)p.empty_out());
        show("empty:");
    }
    {
        Pool p;
        p.put(space(3, 0), 100);
        context_of[0] = 10;
        std::printf("%d ", (int)p.empty_out());
        show("nothing to free:");
    }
    {
        Pool p;
        for (int i = 0; i < 4; ++i) p.put(space(10 + i, i % 2), 100);
        context_of[1] = 11;  // device 1 was reset: 11 and 13 are stale
        p.put(space(14, 0), 100);  // 10 makes room
        show("full, own device:");
        p.put(space(15, 0), 100);  // the other device's 11 makes room
        show("full, the other device's is stale:");
        std::printf("taken %d", take(p, 1));
        std::printf(" %d\n", take(p, 0));
        context_of[0] = 0;  // no context at all
        std::printf("taken %d\n", take(p, 0));
        std::printf("%d ", (int)p.empty_out());
        show("no context:");
    }
    context_of = {{0, 7}, {1, 9}};
    {
        Pool p;
        p.put(space(20, 0, 30), 100);
        p.put(space(21, 0, 50), 100);
        p.put(space(22, 1, 90), 100);
        p.put(space(23, 0, 40), 100);  // 30 + 50 + 40 > 100
        show("bytes:");
        p.put(space(24, 0, 101), 100);  // above the limit by itself
        show("too large:");
        context_of[0] = 12;
        p.put(space(25, 0, 10), 100);  // 21 and 23 are stale
        show("stale ones of the device:");
        std::printf("taken %d", take(p, 0));
        std::printf(" %d", take(p, 0));
        std::printf(" %d\n", take(p, 1));
    }
}
"""

EXPECTED = """\
1 emptied after a reset: freed 2 forgotten 1
0 empty: freed forgotten
0 nothing to free: freed forgotten 3
full, own device: freed 10 forgotten
full, the other device's is stale: freed forgotten 11
taken -1 12
taken -1
0 no context: freed forgotten 13 14 15
bytes: freed 20 forgotten
too large: freed 24 forgotten
stale ones of the device: freed forgotten 21 23
taken 25 -1 22
"""


def test_policy(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe), "-lpthread"],
                   check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == EXPECTED


RESET = r"""
import ctypes, glob, importlib, os, sys
sys.path.insert(0, %r)
nb = importlib.import_module("necsim-rust_b200")
def call(n=40):
    o = nb.simulate(0.01, nb.NonSpatial((n, 30), 2), 5)
    return (o.steps, o.biodiversity, o.speciation.tobytes())
def too_large():
    # 60,000 * 60,000 lineages: its one allocation is refused
    try:
        nb.simulate(0.01, nb.NonSpatial((60000, 60000), 1), 5)
    except nb.NecsimError as e:
        return e.code
first = [call(), call(50)]
assert too_large() == %d       # frees the two kept workspaces
assert [call(), call(50)] == first
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuDevicePrimaryCtxReset_v2(0) == 0
code = too_large()             # forgets the two kept workspaces
print("after the reset:", code)
print("same", [call(), call(50)] == first)
"""


@pytest.mark.gpu
def test_context_reset_between_calls():
    r = subprocess.run([sys.executable, "-c", RESET % (ROOT, -3)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split("\n")[:2] == ["after the reset: -3", "same True"]
