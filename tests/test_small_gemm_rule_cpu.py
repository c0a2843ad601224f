"""CPU test of the rule that sends a plain product to small tiles
(small_gemm_cfg, gemm_small.cu), compiled for the host: products of short K and
many tiles, which small tiles made up to half as long again, stay on the
128-wide ones, in whatever way the operands are stored; those that small tiles
made two to three times faster keep them."""
from __future__ import annotations

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rblas_b200", "csrc")

HOST = r"""
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
struct SmallOperands { bool a_k, b_k, a_vec, b_vec; };
static bool simt_narrow_f32(size_t m, size_t n) {
    const size_t tm = (m + 127) / 128, wide = tm * ((n + 127) / 128), narrow = tm * ((n + 63) / 64);
    return wide < 148 && 4 * narrow >= 3 * 148;
}
%s
int main(int, char** v) {  // type m n k splits a_k b_k a_vec b_vec
    int x[9];
    for (int i = 1; i < 9; ++i) x[i] = atoi(v[i + 1]);
    const SmallOperands op{x[5] != 0, x[6] != 0, x[7] != 0, x[8] != 0};
    std::printf("%%d\n", v[1][0] == 'f' ? small_gemm_cfg<float>(x[1], x[2], x[3], x[4], 148, op)
                                       : small_gemm_cfg<double>(x[1], x[2], x[3], x[4], 148, op));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    with open(os.path.join(CSRC, "gemm_small.cu")) as f:
        src = f.read()
    start = src.index("template <typename T>\nint small_gemm_cfg(")
    d = tmp_path_factory.mktemp("rule")
    (d / "r.cpp").write_text(HOST % src[start:src.index("\n}\n", start) + 2])
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(d / "r"), str(d / "r.cpp")], check=True)
    return lambda *a: int(subprocess.run([str(d / "r"), *map(str, a)], capture_output=True, text=True, check=True).stdout)


# measured, us: wide -> small 8.3 -> 11.9, 21.7 -> 30.6, 28.8 -> 35, 12.4 -> 18.5, 24.7 -> 30.5
@pytest.mark.parametrize("dt,m,k,a_k,b_k", [("f", 1200, 32, 1, 0), ("f", 2400, 8, 1, 0), ("f", 3000, 16, 1, 0),
                                            ("d", 1700, 16, 1, 1), ("d", 1200, 128, 1, 1)])
def test_short_k_stays_on_wide_tiles(rule, dt, m, k, a_k, b_k):
    assert rule(dt, m, m, k, 1, a_k, b_k, 1, 1) == 0


@pytest.mark.parametrize("dt,m,n,k,splits", [("f", 256, 256, 256, 1), ("f", 512, 512, 512, 1), ("f", 640, 480, 1344, 2),
                                             ("f", 2, 10, 2320, 4), ("d", 256, 256, 256, 1), ("d", 512, 512, 512, 2)])
@pytest.mark.parametrize("a_k", [0, 1])
@pytest.mark.parametrize("b_k", [0, 1])
@pytest.mark.parametrize("vec", [0, 1])
def test_small_products_keep_small_tiles(rule, dt, m, n, k, splits, a_k, b_k, vec):
    assert rule(dt, m, n, k, splits, a_k, b_k, vec, vec) > 0
    if dt == "f":
        assert rule(dt, 768, 768, 768, 1, a_k, b_k, vec, vec) == 2
