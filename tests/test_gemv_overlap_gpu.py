"""GPU test of gemv with y in x's memory or in A's: every sum is taken before y
is written, so the result is that of the same call on separate copies, bit for
bit -- in one range and in several, few and many columns, each direction."""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import complex2, level2
from rblas_b200.types import Layout, Transpose

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
@pytest.mark.parametrize("trans", [Transpose.NoTrans, Transpose.Trans])
@pytest.mark.parametrize("m,n", [(31, 31), (1000, 20), (700, 700), (5000, 40), (40, 5000), (1024, 4800), (3000, 1500)])
def test_overlapping_vectors(dt, trans, m, n):
    tdt, ndt = getattr(torch, dt), np.dtype(dt)
    g = torch.Generator(device="cuda")
    g.manual_seed(m + 5 * n)
    a = torch.randn(m * n, dtype=tdt, device="cuda", generator=g)
    lx, ly = (n, m) if trans == Transpose.NoTrans else (m, n)
    v = torch.randn(lx + ly, dtype=tdt, device="cuda", generator=g)
    gemv = (complex2 if tdt.is_complex else level2).gemv_dev
    el = v.element_size()

    def call(a_ptr, x_ptr, y_ptr):
        gemv(Layout.ColMajor, trans, m, n, 1.25, a_ptr, m, x_ptr, 1, 0.5, y_ptr, 1, ndt,
             stream=torch.cuda.current_stream().cuda_stream)

    for xo, yo in ((0, 0), (0, min(lx, ly) // 2), (ly // 3, 0)):  # x and y share all or part of v
        x, y, both = v[xo:xo + lx].clone(), v[yo:yo + ly].clone(), v.clone()
        call(a.data_ptr(), x.data_ptr(), y.data_ptr())
        call(a.data_ptr(), both.data_ptr() + xo * el, both.data_ptr() + yo * el)
        assert torch.equal(both[yo:yo + ly], y), (xo, yo)
    # y is the head of A
    x, y, mat = v[:lx].clone(), a[:ly].clone(), a.clone()
    call(a.data_ptr(), x.data_ptr(), y.data_ptr())
    call(mat.data_ptr(), x.data_ptr(), mat.data_ptr())
    assert torch.equal(mat[:ly], y)
    assert torch.equal(mat[ly:], a[ly:])
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
