"""The buffers a device's sorts keep, driven with a host allocator that can fail:
they never claim to hold more than was allocated."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "fe_sort_scratch.h"
using namespace fe;
std::map<void*, size_t> live;
int countdown = 0;
int take(void** p, size_t bytes) {
    if (countdown && --countdown == 0) return 2;
    *p = malloc(bytes);
    live[*p] = bytes;
    return 0;
}
void give(void* p) {
    if (p && live.erase(p) != 1) { printf("freed twice\n"); exit(1); }
    free(p);
}
size_t size(void* p) { return live.count(p) ? live[p] : 0; }
int main() {
    for (int k = 1; k <= 3; ++k) {
        SortBuffers S;
        // a sort, a larger one whose k-th allocation fails, a small one (its error
        // word alone), then sorts of every size
        const struct { uint32_t n; size_t words; int fail; } calls[] = {
            {1000, 50, 0}, {2000, 90, k}, {1000, 50, 0}, {10, 90, 0}, {2000, 10, 0}, {1, 1, 0}};
        for (auto c : calls) {
            if (!S.flags) take((void**)&S.flags, kSortFlagWords * 4);
            if (sort_buffers_hold(S, c.n, c.words)) goto check;
            countdown = c.fail;
            if (int e = sort_buffers_grow(S, c.n, c.words, take, give)) {
                if (!c.fail || e != 2) { printf("unexpected failure\n"); return 1; }
                if (size(S.flags) < kSortFlagWords * 4) { printf("error word lost\n"); return 1; }
                continue;
            }
            if (c.fail) { printf("failure not reported\n"); return 1; }
        check:
            if (size(S.tk) < c.n * 4 || size(S.tv) < c.n * 4 || size(S.words) < c.words * 4) {
                printf("k %d: n %u words %zu do not fit\n", k, c.n, c.words);
                return 1;
            }
        }
        give(S.tk); give(S.tv); give(S.words); give(S.flags);
        if (!live.empty()) { printf("leak\n"); return 1; }
    }
    return 0;
}
"""


def test_buffers_after_a_failed_growth(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "fluid-engine_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
