"""Host: memory taken all or none, and arrays that grow (csrc/mp_alloc.h), with an
allocator that fails at each of its calls in turn: no pointer and no length is
left set, nothing is left allocated and nothing is freed twice."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "mini-fem-pic-main_b200", "csrc")

PROGRAM = r"""
#include <cstdlib>
#include <set>
#include "mp_alloc.h"

static std::set<void *> live;
static int calls, fail_at;
static bool take(void **p, size_t bytes) {
    if (calls++ == fail_at) {
        *p = reinterpret_cast<void *>(64);  // as a failing call may leave it
        return false;
    }
    live.insert(*p = std::malloc(bytes));
    return true;
}
static void give(void *p) {
    if (!live.erase(p)) std::exit(1);
    std::free(p);
}

int main() {
    for (fail_at = 0; fail_at < 4; fail_at++) {
        void *a = &a, *b = &b, *c = &c;
        calls = 0;
        const bool ok = mp::allocate_all({{&a, 16}, {&b, 32}, {&c, 48}}, take, give);
        if (ok != (fail_at == 3)) return 2;
        if (ok ? live.size() != 3 || !a || !b || !c : !live.empty() || a || b || c) return 3;
    }
    for (void *p : std::set<void *>(live)) give(p);
    // an array grows, fails to, and is asked for less than it held before
    int *p = nullptr;
    long long len = 0;
    calls = 0;
    fail_at = 1;
    if (!mp::grow(p, len, 10, 20, take, give) || len != 20 || live.count(p) != 1) return 4;
    if (!mp::grow(p, len, 20, 40, take, give) || len != 20 || calls != 1) return 5;
    if (mp::grow(p, len, 21, 42, take, give) || p || len || !live.empty()) return 6;
    if (!mp::grow(p, len, 5, 10, take, give) || len != 10 || live.size() != 1) return 7;
    return 0;
}
"""


def test_all_or_none(tmp_path):
    src, exe = tmp_path / "a.cpp", tmp_path / "a"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
