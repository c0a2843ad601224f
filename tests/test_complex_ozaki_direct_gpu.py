"""GPU test of the complex GEMM in the INT8-slice form, whose passes over A
read the complex matrix itself: equal, bit for bit, to the real GEMM in that
form on A's real form [[Re, -Im], [Im, Re]] written out, for every op(A), at
the edges of the passes' tiles (32 complex elements a side, 1024 columns of K),
with a zero row, infinities and NaNs. The form itself is checked against the
oracle elsewhere.
"""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import complex3, level3
from rblas_b200.types import Layout, Precision, Transpose

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ta", ["n", "t", "c"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 17, 31), (64, 40, 65), (130, 70, 1025), (257, 33, 96)])
def test_direct_matches_real_form(m, n, k, ta):
    g = torch.Generator(device="cuda")
    g.manual_seed(m * 31 + k)
    rows, cols = (m, k) if ta == "n" else (k, m)
    lda = rows + 3
    A = torch.randn(cols, lda, dtype=torch.complex128, device="cuda", generator=g)  # column-major: [col, row]
    A *= torch.exp2(torch.randint(-40, 40, (cols, lda), device="cuda", generator=g).double())
    B = torch.randn(n, k, dtype=torch.complex128, device="cuda", generator=g)
    op = A[:, :rows].T if ta == "n" else A[:, :rows]
    for special in (False, True):
        if special:
            op[m // 2] = 0
            op[0, k - 1] = complex(float("inf"), 1.0)
            op[m - 1, 0] = complex(2.0, float("nan"))
        oa = op.conj().resolve_conj() if ta == "c" else op
        real = torch.empty(k, 2, m, 2, dtype=torch.float64, device="cuda")  # column-major 2m x 2k
        real[:, 0, :, 0], real[:, 0, :, 1] = oa.real.T, oa.imag.T
        real[:, 1, :, 0], real[:, 1, :, 1] = 0.0 - oa.imag.T, oa.real.T
        C = torch.full((n, m), float("nan"), dtype=torch.complex128, device="cuda")
        P = torch.empty(n, m, 2, dtype=torch.float64, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        complex3.gemm_dev({"n": Transpose.NoTrans, "t": Transpose.Trans, "c": Transpose.ConjTrans}[ta], Transpose.NoTrans,
                          m, n, k, 1.0, A.data_ptr(), lda, B.data_ptr(), k, 0.0, C.data_ptr(), m, np.complex128,
                          prec=Precision.Ozaki, stream=st)
        level3.gemm_dev(Layout.ColMajor, Transpose.NoTrans, Transpose.NoTrans, 2 * m, n, 2 * k, 1.0, real.data_ptr(), 2 * m,
                        B.data_ptr(), 2 * k, 0.0, P.data_ptr(), 2 * m, np.float64, prec=Precision.Ozaki, stream=st)
        torch.cuda.synchronize()
        want = torch.stack([P[..., 0] + (0.0 - 0.0 * P[..., 1]), P[..., 1] + 0.0 * P[..., 0]], -1)  # 1 * P, complex
        assert torch.allclose(torch.view_as_real(C), want, rtol=0, atol=0, equal_nan=True)
    assert rb.device_error()[0] == 0
