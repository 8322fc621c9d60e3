"""CPU: the fold of a query CTA's replicated cells into the accumulators, taken
from the generated source and run by host threads, for CTAs of any number of
threads (whole warps or not)."""
import os
import re
import shutil
import subprocess

import pytest

from ultraprecise_b200 import abi, prewarm
from ultraprecise_b200 import expr as E

HERE = os.path.dirname(os.path.abspath(__file__))

HARNESS = r"""
#include <barrier>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <thread>
#include <vector>
typedef uint32_t u32; typedef uint64_t u64; typedef int64_t i64;
#define UP_DI static inline
struct Dim { unsigned x; };
static thread_local Dim threadIdx, blockDim;
static std::barrier<>* bar;
static void __syncthreads() { bar->arrive_and_wait(); }
static u32 atomicAdd(u32* p, u32 v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
static u64 atomicAdd(u64* p, u64 v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
struct UpQArgs { u32* acc; u64* cnt; };
"""

MAIN = r"""
int main() {
    std::mt19937_64 rng(7);
    constexpr int S = 64;
    for (int T : {1, 7, 16, 31, 32, 48, 64}) for (int rep : {1, 2, 8, 32}) for (int ng : {1, 2, 7}) {
        if (ng * rep > S) continue;
        std::vector<int> cells(WP * S, 0);
        std::vector<__int128> sum(ng, 0);
        std::vector<u64> rows(ng, 0);
        for (int g = 0; g < ng; g++) for (int r = 0; r < rep; r++) {
            for (int w = 0; w < WP - 1; w++) {
                const int v = (int)(rng() % 4000001) - 2000000;
                cells[w * S + g * rep + r] = v;
                sum[g] += (__int128)v << (16 * w);
            }
            const int n = (int)(rng() % 1000);
            cells[(WP - 1) * S + g * rep + r] = n;
            rows[g] += n;
        }
        std::vector<u32> acc(ng * W, 0);
        std::vector<u64> cnt(ng, 0);
        UpQArgs a{acc.data(), cnt.data()};
        std::barrier<> b(T);
        bar = &b;
        std::vector<std::thread> th;
        for (int t = 0; t < T; t++) th.emplace_back([&, t] {
            threadIdx.x = t; blockDim.x = T;
            q_cells_flush<S>(a, cells.data(), ng, rep);
        });
        for (auto& t : th) t.join();
        for (int g = 0; g < ng; g++) {
            __int128 v = 0;
            std::memcpy(&v, &acc[g * W], 4 * W);
            if (acc[g * W + W - 1] >> 31) for (int i = W; i < 4; i++) v |= (__int128)0xffffffffu << (32 * i);
            if (v != sum[g] || cnt[g] != rows[g]) { std::printf("T=%d rep=%d ng=%d g=%d\n", T, rep, ng, g); return 1; }
        }
        for (int c : cells) if (c) { std::printf("T=%d rep=%d ng=%d: a cell is left\n", T, rep, ng); return 1; }
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_cells_are_folded_by_any_number_of_threads(tmp_path):
    src = prewarm.query_source([E.col(0)], [E.ColType(12, 2)], [(abi.UP_AGG_SUM, 0)])
    flush = re.search(r"template <int S>\nUP_DI void q_cells_flush\(.*?\n}\n", src, re.S).group(0)
    dev = open(os.path.join(HERE, os.pardir, "ultraprecise_b200", "csrc", "up_dev.cuh")).read()
    parts = [re.search(r"template <[^>]*>\nUP_DI \w+ " + name + r"\(.*?\n}\n", dev, re.S).group(0)
             for name in ("atomic_add_twos", "cells_limb", "fold_limbs")]
    wp = int(re.search(r"constexpr int WP = (\d+);", flush).group(1))
    words = int(re.search(r"a\.acc \+ \(i64\)g \* (\d+) \+ 0, t\)", flush).group(1))
    cpp, exe = str(tmp_path / "cells.cpp"), str(tmp_path / "cells")
    with open(cpp, "w") as f:
        f.write(HARNESS + "".join(parts) + flush + f"constexpr int WP = {wp}, W = {words};\n" + MAIN)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-o", exe, cpp], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_cells_fit_the_ctas_they_are_planned_for():
    """Slots and pieces of the cell kernels, over widths and numbers of sums:
    the first kernel's within 40 KB, the second's within one of two CTAs of an
    SM beside the input stages, and never fewer than the first's."""
    import random
    rng = random.Random(2)
    second = 0
    for _ in range(200):
        n = rng.randint(1, 10)
        types = [E.ColType(rng.randint(1, 80), 0) for _ in range(3)]
        a, b, c = (E.col(i) for i in range(3))
        exprs = [rng.choice([a * b, a, b - c, a * b * c, a + c]) for _ in range(n)]
        src = prewarm.query_source(exprs, types, [(abi.UP_AGG_SUM, i) for i in range(n)])
        inst = [tuple(map(int, m)) for m in re.findall(r"up_query_cells_body<(\d+), (\d+), (\d+), (\d+)>\(a, sm\)", src)]
        if not inst:
            continue
        wp = int(re.search(r"constexpr int R = \d+, WP = (\d+), NLS", src).group(1))
        tags = int(re.search(r"int\* tags = \(int\*\)\(sm \+ (\d+)\);", src).group(1))
        s, h, _, gmax = inst[0]
        assert s == h == gmax and (s == 4 or wp * s * 4 <= 40 * 1024)
        if len(inst) == 2:
            s2, h2, gmin, gmax2 = inst[1]
            second += 1
            assert s2 == gmax2 > s and h2 == 0 and gmin >= s
            assert tags + wp * s2 * 4 + 32 <= 113 * 1024
    assert second > 50
