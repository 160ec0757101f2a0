"""The chunk-end exchange of one warp, run on the host lane by lane: a shuffle or a warp reduction lets a lane run on without
the others' writes, only __syncwarp() holds it back.  Whatever order the lanes take, the slots, their inverse, the rewritten
samples and the counts are those of one thread walking the pairs, on the energies that the last replica's arrival makes
visible."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

SRC = r"""
#include <ucontext.h>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <numeric>
#include <random>
#include <vector>

// the warp: a lane runs until it waits at __syncwarp() (or, lane 0, for the other lanes' terms of a sum); then the next lane
// of the order runs
static ucontext_t home, ctx[32];
static std::vector<char> stack[32];
static std::function<void(int)> body;
static int cur, terms, sum;
static bool done[32], waits[32], wait_sum;
static std::function<void()> arrival;
static void yield() { swapcontext(&ctx[cur], &home); }
static void __syncwarp() { waits[cur] = true; yield(); }
static void __threadfence() {}
static int __shfl_sync(unsigned, int v, int) { return cur == 0 ? v : 1; }      // (the replica that arrives last)
static int __reduce_add_sync(unsigned, int v) {                               // (only lane 0 uses the sum)
    sum += v; ++terms;
    if (cur == 0 && terms < 32) { wait_sum = true; yield(); wait_sum = false; }
    return cur == 0 ? sum : 0;
}
static int atomicAdd(int *p, int v) { const int x = *p; *p += v; arrival(); return x; }
template <typename T> static T __ldcg(const T *p) { return *p; }
static void entry(int lane) { body(lane); done[lane] = true; yield(); }

#include "ce_exchange.cuh"
using namespace nce;

static void warp(const std::vector<int> &order) {
    terms = sum = 0; wait_sum = false;
    for (int l = 0; l < 32; ++l) {
        done[l] = waits[l] = false;
        stack[l].resize(1 << 16);
        getcontext(&ctx[l]);
        ctx[l].uc_stack.ss_sp = stack[l].data(); ctx[l].uc_stack.ss_size = stack[l].size(); ctx[l].uc_link = &home;
        makecontext(&ctx[l], (void (*)())entry, 1, l);
    }
    for (;;) {
        int next = -1, held = 0;
        for (int l : order) {
            if (done[l]) continue;
            if (waits[l]) { ++held; continue; }
            if (l == 0 && wait_sum && terms < 32) continue;
            next = l; break;
        }
        if (next < 0 && !held) return;
        if (next < 0) { for (int l = 0; l < 32; ++l) { if (!done[l] && !waits[l]) { std::puts("stuck"); std::exit(2); } waits[l] = false; } continue; }
        cur = next;
        swapcontext(&home, &ctx[next]);
    }
}

struct Job {
    int32_t R; double *E; const float *beta_slot; int32_t *rep_of_slot, *slot_of_rep; const int32_t *ladder_id; int64_t *n_ex;
    uint64_t seed; const double *ex_u; int32_t *ex_sync, ex_flags; const int64_t *step_dev; int64_t n_steps, sample_interval;
    double *E_samples;
};

int main() {
    std::mt19937 g(7);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    for (int R : {2, 3, 31, 32, 33, 64, 65, 66, 131, 300})
        for (int kind = 0; kind < 12; ++kind) {
            const int rounds = kind < 8 ? 1 : 3;                 // several rounds: exchange_warp alone
            std::vector<int32_t> ros(R), sor(R), lid(R);
            std::vector<float> beta(R);
            std::vector<double> E(R), old(R), u((size_t)rounds * (R / 2)), Es((size_t)2 * R, -1.0);
            std::iota(ros.begin(), ros.end(), 0); std::shuffle(ros.begin(), ros.end(), g);
            for (int i = 0; i < R; ++i) { sor[ros[i]] = i; lid[i] = 3 * i / (R + 1); beta[i] = (float)(1.0 + 0.1 * i); E[i] = U(g); old[i] = -1e6 * U(g); }
            for (auto &x : u) x = U(g);
            const int par = kind & 7;
            std::vector<int32_t> want(ros);                      // one thread
            int64_t n = 0;
            for (int q = 0; q < rounds; ++q) {
                const std::vector<int32_t> was(want);
                for (int k = 0; 2 * k < R - 1; ++k) {
                    const int a = 2 * k + ((par >> q) & 1), b = a + 1;
                    if (b >= R || lid[a] != lid[b]) continue;
                    if (std::log(u[(size_t)q * (R / 2) + k]) < ((double)beta[b] - (double)beta[a]) * (E[was[b]] - E[was[a]])) { std::swap(want[a], want[b]); ++n; }
                }
            }
            std::vector<int> order(32);
            for (int l = 0; l < 32; ++l) order[l] = kind % 4 == 0 ? 31 - l : l;
            if (kind % 4 > 1) std::shuffle(order.begin(), order.end(), g);
            int64_t n_ex = 5, step = 0;
            int32_t sync = R - 1;
            std::vector<double> seen(old);                       // what the lanes read until lane 0 has seen every replica arrive
            if (rounds == 1) {
                Job jb = {R, seen.data(), beta.data(), ros.data(), sor.data(), lid.data(), &n_ex, 1, u.data(), &sync, 1 | (par & 1) << 1, &step, 20, 10, Es.data()};
                arrival = [&] { seen = E; jb.E = seen.data(); };
                body = [&](int lane) { fused_chunk_end(jb, 0, lane); };
                warp(order);
                if (step != 20 || sync != 0) { std::printf("R %d: step %lld sync %d\n", R, (long long)step, sync); return 1; }
            } else {
                ExArgs x = {R, E.data(), 1.0, beta.data(), ros.data(), sor.data(), lid.data(), &n_ex, 1, 0, u.data(), par, rounds, Es.data(), 1};
                body = [&](int lane) { exchange_warp(x, lane); };
                warp(order);
            }
            if (ros != want || n_ex != 5 + n) { std::printf("R %d kind %d: slots differ\n", R, kind); return 1; }
            for (int i = 0; i < R; ++i)
                if (sor[want[i]] != i || Es[R + i] != E[want[i]] || Es[i] != -1.0) { std::printf("R %d kind %d: slot %d stale\n", R, kind, i); return 1; }
        }
    std::puts("ok");
    return 0;
}
"""


def test_any_order_of_lanes(tmp_path):
    cxx = shutil.which("g++") or pytest.skip("no C++ compiler")
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if p and os.path.exists(f"{p}/include/cuda_runtime.h")), None)
    if cuda is None:
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "warp.cpp", tmp_path / "warp"
    src.write_text(SRC)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "neuralce_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-I", f"{cuda}/include", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout)
