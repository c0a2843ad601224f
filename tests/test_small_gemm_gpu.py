"""GPU test of the plain GEMM on small tiles: at the edges of its tiles and
stages, with operands on and off 16 bytes, every layout of op(A) and op(B),
the result equals the grouped kernel's on 128-wide tiles bit for bit (each
element's sum runs over k in the same order, in the ranges that one splits K
into where it does), infinities and NaNs included. The grouped kernel is checked against the
oracle in test_serving_gpu.py."""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import level3, serving
from rblas_b200.types import Layout, Transpose

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("ta", [Transpose.NoTrans, Transpose.Trans])
@pytest.mark.parametrize("tb", [Transpose.NoTrans, Transpose.Trans])
@pytest.mark.parametrize("pad,off", [(0, 0), (4, 0), (1, 0), (0, 1)])
def test_small_tiles(dt, ta, tb, pad, off):
    tdt = torch.float32 if dt == np.float32 else torch.float64
    g = torch.Generator(device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    for m, n, k, beta in ((1, 1, 1, 0.0), (31, 33, 7, 1.0), (32, 32, 32, -0.5), (33, 65, 31, 0.5), (64, 64, 97, 1.0), (127, 129, 33, 0.0),
                          (300, 200, 400, -0.5), (513, 500, 300, 1.0), (700, 640, 250, 0.5), (17, 2001, 64, 1.0), (3001, 5, 129, 0.5),
                          (250, 190, 1100, 0.5), (512, 512, 530, 1.0), (100, 90, 2051, 0.5)):
        g.manual_seed(m * 7 + n * 3 + k)
        ar, ac = (m, k) if ta == Transpose.NoTrans else (k, m)
        br, bc = (k, n) if tb == Transpose.NoTrans else (n, k)
        lda, ldb, ldc = ar + pad, br + pad, m + pad
        a, b, c0 = (torch.randn(off + ld * c, dtype=tdt, device="cuda", generator=g)[off:] for ld, c in ((lda, ac), (ldb, bc), (ldc, n)))
        for special in (False, True):
            if special:
                a[a.numel() // 2] = float("inf")
                b[b.numel() // 3] = float("nan")
            one, many = c0.clone(), c0.clone()
            level3.gemm_dev(Layout.ColMajor, ta, tb, m, n, k, 1.5, a.data_ptr(), lda, b.data_ptr(), ldb, beta, one.data_ptr(), ldc, dt,
                            stream=st)
            p = serving.Problem(dt, Layout.ColMajor, ta, tb, m, n, k, 1.5, a.data_ptr(), lda, b.data_ptr(), ldb, beta, many.data_ptr(), ldc)
            serving.grouped_gemm([p], stream=st)
            assert torch.equal(torch.isnan(one), torch.isnan(many)), (m, n, k)
            assert torch.equal(one.nan_to_num(7.0), many.nan_to_num(7.0)), (m, n, k)
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
