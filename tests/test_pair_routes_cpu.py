"""CPU test: the shapes that the GPU tests of the CTA-pair kernels use run on
those kernels. The dispatch rules (gemm_umma.cu) are compiled for the host and
asked for a B200's 148 SMs."""
from __future__ import annotations

import ast
import os
import subprocess

import pytest

TESTS = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(TESTS), "rblas_b200", "csrc")

HOST = r"""
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>
#define __host__
#define __device__
#define __forceinline__ inline
constexpr int kOzGroups = 3, kPzN = 128, kPzTileElems = 256 * kPzN;
struct OzParams {
    int num_tiles, num_kt, slices, kchunks, tail_tiles, parts[kOzGroups], order[kOzGroups], plane0[kOzGroups], planes;
};
%s
// m n k slices -> Ozaki pairs, tail tiles, parts of the dearest group, BF16 pairs (3x, X6), tall form
int main(int, char** v) {
    const int m = atoi(v[1]), n = atoi(v[2]), k = atoi(v[3]), slices = atoi(v[4]);
    OzParams p{};
    p.num_tiles = ((m + 255) / 256) * ((n + 127) / 128);
    p.num_kt = (k + 127) / 128;
    p.slices = slices;
    const int per = static_cast<int>(std::max(2147483647LL / (static_cast<long long>(slices) * 128 * 128) / 128, 1LL));
    p.kchunks = (p.num_kt + per - 1) / per;
    ozaki_pair_tail(p, 74);
    std::printf("%%d %%d %%d %%d %%d %%d %%d\n", ozaki_pair_tiles(m, n), p.tail_tiles,
                p.tail_tiles ? *std::max_element(p.parts, p.parts + kOzGroups) : 0, p.kchunks, bf16_pair_tiles(2, m, n, 148),
                bf16_pair_tiles(3, m, n, 148), bf16_fused_a(false, n, nullptr, m));
}
"""


@pytest.fixture(scope="module")
def route(tmp_path_factory):
    with open(os.path.join(CSRC, "gemm_umma.cu")) as f:
        src = f.read()
    names = ("__host__ __device__ __forceinline__ int pz_nd(", "double ozaki_pair_tail_load(", "void ozaki_pair_tail(",
             "bool ozaki_pair_tiles(", "bool bf16_pair_tiles(", "bool bf16_fused_a(")
    parts = []
    for name in names:
        start = src.index(name)
        line = src.index("\n", start)
        parts.append(src[start:line] if src[line - 1] == "}" else src[start:src.index("\n}\n", start) + 2])
    d = tmp_path_factory.mktemp("routes")
    (d / "r.cpp").write_text(HOST % "\n".join(parts))
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(d / "r"), str(d / "r.cpp")], check=True)

    def ask(m, n, k, slices=8):
        out = subprocess.run([str(d / "r"), *map(str, (m, n, k, slices))], capture_output=True, text=True, check=True).stdout
        return dict(zip(("ozaki", "tail", "parts", "chunks", "x3", "x6", "tall"), map(int, out.split())))

    return ask


@pytest.fixture(scope="module")
def shapes():
    with open(os.path.join(TESTS, "test_pair_padding_gpu.py")) as f:
        tree = ast.parse(f.read())
    return {s.targets[0].id: ast.literal_eval(s.value) for s in tree.body
            if isinstance(s, ast.Assign) and s.targets[0].id in ("OZ_WHOLE", "OZ_TAIL", "OZ_SLICES", "BF16", "TALL")}


def test_ozaki_routes(route, shapes):
    for s in shapes["OZ_WHOLE"]:
        assert route(*s)["ozaki"] and not route(*s)["tail"], s
    assert any(route(*s)["chunks"] > 1 for s in shapes["OZ_WHOLE"])
    for s in shapes["OZ_TAIL"]:
        assert route(*s)["ozaki"] and route(*s)["parts"] > 1, s
    for slices in range(2, 13):
        r = route(*shapes["OZ_SLICES"], slices)
        assert r["ozaki"] and r["parts"] > 1, slices


def test_bf16_routes(route, shapes):
    for s in shapes["BF16"]:
        assert route(*s)["x3"] and route(*s)["x6"], s
    ks = [s[2] for s in shapes["BF16"]]
    assert any(k > 2 * 64 and k % 64 for k in ks)  # several units, the last one short
    for s in shapes["TALL"]:
        assert s[0] % 4 == 0, s
        assert route(*s)["tall"] == 1, s
