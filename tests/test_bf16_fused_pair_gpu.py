"""GPU test of the BF16-split GEMM that splits A on CTA pairs (tall products,
A's rows contiguous): the rings, the two splitter groups and the pair's tiles
at their edges -- odd numbers of K tiles over several tiles of a pair, a last
unit of one K tile, a pair whose second half has no rows, one and two column
tiles -- equal the two-pass form (the same matrix stored transposed) bit for
bit, infinities and NaNs included. That form is checked against the oracle in
test_precision_gpu.py.
"""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import level3
from rblas_b200.types import Layout, Precision

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", [Precision.Bf16x3, Precision.Bf16x6])
@pytest.mark.parametrize("m,n,k", [(4, 1, 1), (128, 17, 65), (260, 129, 192), (40000, 30, 64), (40004, 128, 129),
                                   (20000, 256, 321), (57000, 7, 193)])
def test_fused_pair_matches_two_pass(form, m, n, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(m + 3 * n + 7 * k)
    A, B, C0 = (torch.rand(s, dtype=torch.float32, device="cuda", generator=g) * 2 - 1 for s in (m * k, k * n, m * n))
    for special in (False, True):
        if special:
            A[(m * k) // 3], B[(k * n) // 2], C0[m * n - 1] = float("inf"), float("nan"), float("-inf")
        At = A.view(k, m).t().contiguous().view(-1)
        fused, two_pass = C0.clone(), C0.clone()
        level3.gemm_dev(Layout.ColMajor, 0, 0, m, n, k, 1.25, A.data_ptr(), m, B.data_ptr(), k, -0.5, fused.data_ptr(),
                        m, np.float32, prec=form)
        level3.gemm_dev(Layout.ColMajor, 1, 0, m, n, k, 1.25, At.data_ptr(), k, B.data_ptr(), k, -0.5,
                        two_pass.data_ptr(), m, np.float32, prec=form)
        torch.cuda.synchronize()
        assert special or not torch.isnan(fused).any()
        assert torch.allclose(fused, two_pass, rtol=0, atol=0, equal_nan=True)
    assert rb.device_error()[0] == 0
