"""The warp-level ranking of the radix passes (``warp_rank`` in ``common.cuh``) run on the CPU, lane by lane: the
function's own source is compiled for the host with the warp intrinsics as meeting points of 32 fibers, and between two
meeting points the lanes run one after another in forward, reverse or shuffled order. CUDA allows any of these orders
(independent thread scheduling), so the ranks have to be stable under all of them."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
COMMON = os.path.join(ROOT, "kolmo_gb300", "csrc", "common.cuh")

HARNESS = r"""
#include <ucontext.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <random>
#include <vector>
typedef uint32_t u32;
typedef uint64_t u64;
#define __device__
#define __forceinline__ inline

static ucontext_t sched, lanes[32];
static std::vector<char> stacks[32];
static bool done[32];
static int cur;
static u32 slot[2][32], seq[32];

static u32 lane_id() { return (u32)cur; }
// A meeting point: the lane waits until the scheduler has run every other lane to the same one.
static void meet() {
    const int me = cur;
    swapcontext(&lanes[me], &sched);
    cur = me;
}
static u32 *exchange(u32 v) {
    u32 *s = slot[seq[cur]++ & 1];
    s[cur] = v;
    meet();
    return s;
}
static u32 __shfl_sync(u32, u32 v, int src) { return exchange(v)[src & 31]; }
static u32 __ballot_sync(u32, bool p) {
    const u32 *s = exchange(p);
    u32 b = 0;
    for (int i = 0; i < 32; i++) b |= s[i] << i;
    return b;
}
static void __syncwarp() { exchange(0); }
static u32 atomicOr(u32 *p, u32 v) { const u32 o = *p; *p |= v; return o; }
static u32 atomicAdd(u32 *p, u32 v) { const u32 o = *p; *p += v; return o; }
static int __popc(u32 v) { return __builtin_popcount(v); }
static int __ffs(u32 v) { return __builtin_ffs((int)v); }

//SOURCE//

constexpr int CALLS = 3;
static u32 digit[CALLS][4][32], got[CALLS][4][32], mask[256 * 4], cnt[256];

template <int Q, bool CHECK>
static void lane_main() {
    for (int c = 0; c < CALLS; c++) {
        u32 d[Q], r[Q];
        for (int q = 0; q < Q; q++) d[q] = digit[c][q][cur];
        warp_rank<Q, CHECK>(mask, cnt, d, r);
        for (int q = 0; q < Q; q++) got[c][q][cur] = r[q];
    }
    done[cur] = true;
}

template <int Q, bool CHECK>
static int run(int order, u32 seed) {
    std::mt19937 rng(seed);
    const int kind = seed % 5;
    for (auto &c : digit)
        for (auto &q : c)
            for (u32 &d : q) {
                d = kind == 0 ? rng() & 255 : kind == 1 ? rng() & 3 : kind == 2 ? 7u : kind == 3 ? 97 + (rng() & 7) : rng() % 24;
                if (CHECK && rng() % 5 == 0) d = 256;
            }
    std::fill(mask, mask + 256 * 4, 0u);
    for (int i = 0; i < 256; i++) cnt[i] = 1000 * i;
    u32 want[256];
    std::copy(cnt, cnt + 256, want);
    int idx[32];
    for (int i = 0; i < 32; i++) {
        idx[i] = order == 1 ? 31 - i : i;
        done[i] = false;
        seq[i] = 0;
        stacks[i].resize(256 << 10);
        getcontext(&lanes[i]);
        lanes[i].uc_stack.ss_sp = stacks[i].data();
        lanes[i].uc_stack.ss_size = stacks[i].size();
        lanes[i].uc_link = &sched;
        makecontext(&lanes[i], (void (*)())lane_main<Q, CHECK>, 0);
    }
    while (!done[0]) {
        if (order == 2) std::shuffle(idx, idx + 32, rng);
        for (int i : idx) { cur = i; swapcontext(&sched, &lanes[i]); }
    }
    for (int i = 0; i < 32; i++) if (!done[i]) return 1;
    for (int c = 0; c < CALLS; c++)
        for (int q = 0; q < Q; q++)
            for (int l = 0; l < 32; l++) {
                const u32 d = digit[c][q][l];
                if (d > 255) continue;
                if (got[c][q][l] != want[d]++) {
                    printf("Q %d order %d seed %u: call %d element %d lane %d digit %u: rank %u, not %u\n", Q, order, seed, c,
                           q, l, d, got[c][q][l], want[d] - 1);
                    return 1;
                }
            }
    for (u32 m : mask) if (m) { printf("mask left set\n"); return 1; }
    return !std::equal(cnt, cnt + 256, want);
}

int main(int argc, char **argv) {
    const int order = atoi(argv[1]);
    for (u32 seed = 0; seed < 40; seed++)
        if (run<4, false>(order, seed) || run<4, true>(order, seed) || run<2, false>(order, seed) ||
            run<2, true>(order, seed))
            return 1;
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    with open(COMMON) as f:
        m = re.search(r"^template <int Q, bool CHECK>\n.*?^}\n", f.read(), re.M | re.S)
    assert m and "warp_rank(" in m.group(0)
    d = tmp_path_factory.mktemp("warp_rank")
    src = d / "warp_rank.cpp"
    src.write_text(HARNESS.replace("//SOURCE//", m.group(0)))
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(d / "warp_rank"), str(src)], check=True)
    return str(d / "warp_rank")


@pytest.mark.parametrize("order", [0, 1, 2], ids=["forward", "reverse", "shuffled"])
def test_ranks_are_stable_in_any_lane_order(harness, order):
    r = subprocess.run([harness, str(order)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
