"""Buffers that belong together (csrc/qkm_alloc.h): with an allocation that fails part way, nothing is left behind and nothing
is lost, so that the next call allocates them all instead of taking the first one for all of them."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "qkm_alloc.h"
#include <cstdio>
#include <cstdlib>

int live = 0, calls = 0;
int main() {
    for (int fail = 0; fail < 4; ++fail) {   // number of the call that fails; 3: none
        void *a = nullptr, *b = nullptr, *c = nullptr;
        const qkm::Want want[] = {{&a, 16}, {&b, 32}, {&c, 48}};
        auto alloc = [&](void** p, size_t n) { if (calls++ == fail) { *p = (void*)1; return 2; } ++live; *p = malloc(n); return 0; };
        auto release = [&](void* p) { --live; free(p); };
        calls = 0;
        const int e = qkm::alloc_all(want, alloc, release);
        std::printf("%d %d %d%d%d %d ", e, live, a != nullptr, b != nullptr, c != nullptr, calls);
        if (e) {   // again, with memory
            calls = 4;
            const int again = qkm::alloc_all(want, alloc, release);
            std::printf("%d %d", again, live);
        }
        std::printf("\n");
        for (const qkm::Want& w : want) release(*w.p);
    }
    return 0;
}
"""


def test_all_or_none(tmp_path):
    src, exe = tmp_path / "alloc.cpp", tmp_path / "alloc"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "qwen-kernel_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert [line.strip() for line in out] == ["2 0 000 1 0 3", "2 0 000 2 0 3", "2 0 000 3 0 3", "0 3 111 3"]
