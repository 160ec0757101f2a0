"""Step bookkeeping of the windowed kernel at both ends of the range of a chunk's steps, run on the host: every step is drawn
once, in order, into a ring slot that no undecided step holds, and the sampled steps are the multiples of the interval --
also at the last steps of the longest chunk (2^31 - 2), where sums of steps pass 2^31.  Signed overflow traps."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

SRC = r"""
#include <cstdio>
#include <initializer_list>
#include <cstdint>
#include "ce_window_steps.cuh"
using namespace nce;
#define OK(c) do { if (!(c)) { std::printf("line %d: T %d si %d s %d\n", __LINE__, T, si, s); return 1; } } while (0)

static uint32_t rng = 1;
static int rnd(int n) { rng = rng * 1664525u + 1013904223u; return (int)((rng >> 8) % (uint32_t)n); }

// windows from step s0 on (every earlier step decided), as the kernel's loop orders them
static int run(int32_t T, int32_t si, int32_t s0) {
    int32_t s = s0, slot[kWinRing];
    for (int i = 0; i < kWinRing; ++i) slot[i] = -1;
    uint32_t drawn = (uint32_t)s0 + 96u;
    for (int i = 0; i < 96 && i < T - s0; ++i) slot[win_slot(s0, i)] = s0 + i;
    int32_t left = si > 0 ? si - s0 % si : 0;
    while (s < T) {
        const int n_w = T - s < 32 ? T - s : 1 + rnd(32);
        for (int i = 0; i < n_w; ++i) OK(slot[win_slot(s, i)] == s + i);
        if (win_draws(drawn, s)) {
            for (int lane = 0; lane < 32; ++lane)
                if (win_in_chunk(drawn, lane, T)) {
                    const int32_t q = (int32_t)drawn + lane;
                    OK(q >= s && q < T && slot[win_slot(q, 0)] < s);
                    slot[win_slot(q, 0)] = q;
                }
            drawn += 32;
        }
        const int limit = 1 + rnd(n_w);
        for (int i = 0; i < 32; ++i) {
            const bool want = si > 0 && i < limit && ((int64_t)s + i + 1) % si == 0;
            OK((si > 0 && left <= limit && win_samples(left, si, i, limit)) == want);
        }
        if (si > 0) left = win_left(left, si, limit);
        s += limit;
        OK(si == 0 || (left >= 1 && left <= si && ((int64_t)s + left) % si == 0));
    }
    return 0;
}

int main() {
    const int32_t top = 2147483646, sis[] = {0, 1, 2, 7, 31, 32, 33, 1000, 1073741824, 1200000000, top - 40, top};
    for (int32_t T : {1, 2, 31, 32, 33, 95, 96, 97, 127, 128, 129, 1000, 5000})
        for (int32_t si : sis)
            for (int k = 0; k < 20; ++k) if (si <= T && run(T, si, 0)) return 1;
    for (int32_t T : {top, top - 1, top - 63, top - 500, 1200000000 + 3})
        for (int32_t si : sis)
            for (int k = 0; k < 20; ++k) if (si <= T && run(T, si, T - 1 - rnd(1200))) return 1;
    std::puts("ok");
    return 0;
}
"""


def test_draws_and_samples(tmp_path):
    cxx = shutil.which("g++") or pytest.skip("no C++ compiler")
    src, exe = tmp_path / "steps.cpp", tmp_path / "steps"
    src.write_text(SRC)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=signed-integer-overflow", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(ROOT, "neuralce_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout)
