"""GPU test of the BF16-split GEMM on CTA pairs (256 x 256 tiles): at shapes
that take it, ragged against its tiles and its K stages, the result equals
the grouped launch's (128 x 128 tiles, the same products in the same order)
bit for bit, infinities and NaNs included. The grouped launch is checked
against the oracle in test_grouped_forms_gpu.py, the single call at 8192^3
in test_precision_gpu.py.
"""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import level3, serving
from rblas_b200.types import Layout, Precision, Transpose

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", [Precision.Bf16x3, Precision.Bf16x6])
@pytest.mark.parametrize("m,n,k,ta,tb", [
    (2048, 2304, 1, "t", "n"), (1921, 2303, 31, "t", "t"), (2047, 2177, 33, "n", "n"), (2048, 2304, 128, "n", "t"),
    (1793, 2305, 129, "t", "n"), (2050, 2300, 481, "t", "n"), (4097, 4609, 97, "n", "n")])
def test_pair_tiles(form, m, n, k, ta, tb):
    g = torch.Generator(device="cuda")
    g.manual_seed(m * 7 + k)
    T = {"n": Transpose.NoTrans, "t": Transpose.Trans}
    A, B, C0 = (torch.rand(s, dtype=torch.float32, device="cuda", generator=g) * 2 - 1 for s in (m * k, n * k, m * n))
    lda, ldb = (m if ta == "n" else k), (k if tb == "n" else n)
    st = torch.cuda.current_stream().cuda_stream

    def single():
        C = C0.clone()
        level3.gemm_dev(Layout.ColMajor, T[ta], T[tb], m, n, k, 1.5, A.data_ptr(), lda, B.data_ptr(), ldb, -0.5, C.data_ptr(), m,
                        np.float32, prec=form, stream=st)
        return C

    def grouped():
        C = C0.clone()
        serving.grouped_gemm_bf16([serving.Problem(np.float32, Layout.ColMajor, T[ta], T[tb], m, n, k, 1.5, A.data_ptr(), lda,
                                                   B.data_ptr(), ldb, -0.5, C.data_ptr(), m)], form, stream=st)
        return C

    assert torch.equal(single().view(torch.int32), grouped().view(torch.int32))
    A[(m * k) // 2] = float("inf")
    B[(n * k) // 3] = float("nan")
    assert torch.equal(single().nan_to_num(7.0), grouped().nan_to_num(7.0))
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
