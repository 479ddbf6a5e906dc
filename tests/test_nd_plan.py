"""Host: the dissection of the sparse direct solve (csrc/mp_nd_plan.cpp) where no
thread can be had: the same plan as with threads, and no exception."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "mini-fem-pic-main_b200", "csrc")

PROGRAM = r"""
#include <cerrno>
#include <dlfcn.h>
#include <pthread.h>
#include <numeric>
#include "mp_nd.h"

static bool none_left;
static int asked;
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    asked++;
    if (none_left) return EAGAIN;
    return reinterpret_cast<decltype(&pthread_create)>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}

int main() {
    // a cube of 22^3 unknowns, each coupled to its 26 neighbours
    const int m = 22, n = m * m * m;
    std::vector<long long> ptr(1, 0), slot;
    std::vector<int> col;
    std::vector<double> pos;
    for (int z = 0; z < m; z++)
        for (int y = 0; y < m; y++)
            for (int x = 0; x < m; x++) {
                for (int k = 0; k < 27; k++) {
                    const int u = x + k % 3 - 1, v = y + k / 3 % 3 - 1, w = z + k / 9 - 1;
                    if (u >= 0 && v >= 0 && w >= 0 && u < m && v < m && w < m) col.push_back(u + m * (v + m * w));
                }
                ptr.push_back((long long)col.size());
                pos.insert(pos.end(), {(double)x, (double)y, (double)z});
            }
    slot.resize(col.size());
    std::iota(slot.begin(), slot.end(), 0ll);
    mp::NdPlan with, without;
    if (!mp::nd_build_plan(n, ptr, col, slot, pos, 1 << 24, with) || !asked) return 2;
    none_left = true;
    asked = 0;
    if (!mp::nd_build_plan(n, ptr, col, slot, pos, 1 << 24, without) || !asked) return 3;
    return with.perm == without.perm && with.tile_row == without.tile_row && with.ent_src == without.ent_src &&
                   with.chain == without.chain && with.products == without.products &&
                   with.task.size() == without.task.size()
               ? 0 : 4;
}
"""


def test_no_thread(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), os.path.join(CSRC, "mp_nd_plan.cpp"), "-o",
                    str(exe), "-pthread", "-ldl"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
