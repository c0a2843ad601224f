"""CPU test of the Ozaki pair kernel's tail plan (gemm_umma.cu), compiled for
the host: the time it gives the fullest pair is that of dealing the items one
by one as the kernel does, over wave remainders, slice counts, K parts and
numbers of pairs, and the plan of a call takes a few microseconds (it runs on
the host before each call's first launch; item by item it took up to 45)."""
from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rblas_b200", "csrc")

HOST = r"""
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <utility>
#include <vector>
#define __host__
#define __device__
#define __forceinline__ inline
constexpr int kOzGroups = 3, kPzN = 128, kPzTileElems = 256 * kPzN;
struct OzParams {
    int num_tiles, num_kt, slices, kchunks, tail_tiles, parts[kOzGroups], order[kOzGroups], plane0[kOzGroups], planes;
};
struct PzWork { const OzParams* p; int t, u_lo, u_hi, tt, kt0, kt1, plane; };
%s
// the items dealt one by one
static double dealt(const OzParams& p, const int (&cost)[kOzGroups], int pairs, double prod_us) {
    const int groups = (p.slices + 3) / 4, fused = p.num_tiles - p.tail_tiles, total = pz_items(p) - fused;
    double load = 0;
    for (int q = 0; q < pairs; ++q) {
        long long products = 0;
        int items = 0;
        for (int j = q; j < total; j += pairs) {
            PzWork w{};
            pz_item(p, pairs, fused + j, w);
            products += static_cast<long long>(cost[groups - 1 - w.u_lo]) * (w.kt1 - w.kt0);
            ++items;
        }
        load = std::max(load, products * prod_us + 3.0 * items);
    }
    return load;
}
int main() {
    double slowest = 0;
    for (int slices = 2; slices <= 12; ++slices)
        for (int pairs : {1, 7, 74})
            for (int tiles = 1; tiles <= 2 * pairs; ++tiles)
                for (int num_kt : {1, 2, 3, 16, 17, 63}) {
                    OzParams p{};
                    p.num_tiles = tiles;
                    p.num_kt = num_kt;
                    p.slices = slices;
                    p.kchunks = 1;
                    double us = 1e9;
                    for (int r = 0; r < 20; ++r) {
                        const auto t0 = std::chrono::steady_clock::now();
                        ozaki_pair_tail(p, pairs);
                        us = std::min(us, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() * 1e6);
                    }
                    slowest = std::max(slowest, us);
                    const int groups = (slices + 3) / 4;
                    int cost[kOzGroups] = {};
                    for (int g = 0; g < groups; ++g)
                        for (int d = 4 * g; d < 4 * g + pz_nd(slices, g); ++d) cost[g] += d + 1;
                    p.tail_tiles = tiles %% pairs;
                    for (int a = 1; a <= num_kt && a <= 13; a += 4)
                        for (int b = 1; b <= num_kt && b <= 13; b += 3)
                            for (int turn = 0; turn < groups; ++turn) {
                                for (int g = 0; g < groups; ++g) {
                                    p.parts[g] = g == 0 ? a : b;
                                    p.order[g] = (g + turn) %% groups;
                                }
                                if (ozaki_pair_tail_load(p, cost, pairs, 0.15) != dealt(p, cost, pairs, 0.15)) {
                                    std::printf("slices %%d pairs %%d tiles %%d kt %%d parts %%d %%d\n", slices, pairs, tiles, num_kt, a, b);
                                    return 1;
                                }
                            }
                }
    std::printf("%%.1f us\n", slowest);
    return slowest < 25 ? 0 : 2;
}
"""


def test_tail_plan(tmp_path):
    with open(os.path.join(CSRC, "gemm_umma.cu")) as f:
        src = f.read()
    names = ("__host__ __device__ __forceinline__ int pz_nd(", "__host__ __device__ __forceinline__ int pz_items(",
             "__host__ __device__ __forceinline__ void pz_item(", "double ozaki_pair_tail_load(", "void ozaki_pair_tail(")
    parts = []
    for name in names:
        start = src.index(name)
        line = src.index("\n", start)
        parts.append(src[start:line] if src[line - 1] == "}" else src[start:src.index("\n}\n", start) + 2])
    cpp = tmp_path / "plan.cpp"
    cpp.write_text(HOST % "\n".join(parts))
    exe = tmp_path / "plan"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(cpp)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
