"""CPU test of the rule that gives batched f64 trsm its slice width
(trsm_wide_slices, trsm_batched.cu), compiled for the host with a B200's 148
SMs: 16-wide slices where 32-wide ones would start a wave for a few CTAs (they
took up to half as long again), 32-wide ones for batches that fill the GPU, the
shapes of their GPU test among them."""
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
#include <cstdio>
#include <cstdlib>
%s
int main(int, char** v) { std::printf("%%d\n", trsm_wide_slices(atoi(v[1]), atoi(v[2]), atoi(v[3]), 148)); }
"""


@pytest.fixture(scope="module")
def wide(tmp_path_factory):
    with open(os.path.join(CSRC, "trsm_batched.cu")) as f:
        src = f.read()
    start = src.index("bool trsm_wide_slices(")
    d = tmp_path_factory.mktemp("slices")
    (d / "r.cpp").write_text(HOST % src[start:src.index("\n}\n", start) + 2])
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(d / "r"), str(d / "r.cpp")], check=True)
    return lambda *a: int(subprocess.run([str(d / "r"), *map(str, a)], capture_output=True, text=True, check=True).stdout)


@pytest.mark.parametrize("q,nrhs,batch", [(600, 48, 75), (600, 100, 40), (400, 48, 75), (200, 100, 40), (600, 48, 150),
                                          (128, 100, 40), (512, 512, 1), (64, 8, 1024), (64, 16, 149)])
def test_16_wide(wide, q, nrhs, batch):
    assert wide(q, nrhs, batch) == 0


def test_32_wide(wide):
    with open(os.path.join(TESTS, "test_trsm_wide_gpu.py")) as f:
        tree = ast.parse(f.read())
    func = next(n for n in tree.body if isinstance(n, ast.FunctionDef))
    cases = next(d.args[1] for d in func.decorator_list if d.args[0].value.startswith("q,"))
    shapes = [[v.value for v in c.elts[:3]] for c in cases.elts]
    assert len(shapes) == 7
    for s in shapes + [[512, 64, 1024], [512, 4096, 1], [256, 100, 300], [512, 64, 149]]:
        assert wide(*s) == 1, s
