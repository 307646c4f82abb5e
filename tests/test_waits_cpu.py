"""The GEMM kernel's record of bounded waits (csrc/qkm_wait.h), walked on the host: a wait that runs out inside a unit ends the
walk at the next unit, which is not read, is reported, and no further wait is begun."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "qkm_wait.h"
#include <cstdio>

// A role of the kernel: takes units until next() ends it, waits three times in each.  fail: number of the wait that runs out.
static int walk(int units, int fail, bool other_lane) {
    qkm::Waits w;
    int begun = 0, read = 0;
    auto one = [&] { return ++begun - 1 != fail; };
    auto any = [&](bool out) { return out || (other_lane && read == 2); };   // a lane beside this one gave up in the second unit
    for (int k = 0; k < units; ++k) {
        if (!w.next(one, any)) break;
        ++read;
        for (int i = 0; i < 3; ++i) w.wait(one);
    }
    std::printf("%d %d %d\n", read, begun, w.out ? 1 : 0);
    return 0;
}
int main() {
    walk(4, -1, false);   // no wait runs out
    walk(4, 2, false);    // one inside the first unit
    walk(4, 4, false);    // the one for the second unit itself
    walk(4, 15, false);   // the last of the last unit
    walk(4, -1, true);
    return 0;
}
"""


def test_waits_are_sticky(tmp_path):
    src, exe = tmp_path / "waits.cpp", tmp_path / "waits"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "qwen-kernel_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    # units read, waits begun, reported
    assert out[:5] == ["4 16 0", "1 3 1", "1 5 1", "4 16 1", "2 9 1"]
