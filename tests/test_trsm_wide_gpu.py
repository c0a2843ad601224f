"""GPU test of the batched f64 trsm on 32-wide slices (batches that fill the
GPU): orders around its 64-row blocks and up to the largest its shared memory
takes, right-hand sides around its slices, every side, uplo, trans and diag,
by the normwise backward error that test_trsm_batched_gpu.py states:
||op(A) X - alpha B||_F / (||A||_F ||X||_F + |alpha| ||B||_F) <= 4 q u for
every member."""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import level3
from rblas_b200.types import Diag, Side, Transpose, Uplo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("side", [Side.Left, Side.Right])
@pytest.mark.parametrize("uplo", [Uplo.Upper, Uplo.Lower])
@pytest.mark.parametrize("trans", [Transpose.NoTrans, Transpose.Trans])
@pytest.mark.parametrize("q,nrhs,batch,diag", [
    (1, 17, 80, Diag.NonUnit), (63, 33, 60, Diag.Unit), (64, 32, 80, Diag.NonUnit), (65, 31, 80, Diag.NonUnit),
    (130, 64, 40, Diag.Unit), (200, 41, 55, Diag.NonUnit), (679, 18, 80, Diag.NonUnit)])
def test_wide_slices(side, uplo, trans, q, nrhs, batch, diag):
    g = torch.Generator(device="cuda")
    g.manual_seed(q * 3 + nrhs)
    m, n = (q, nrhs) if side == Side.Left else (nrhs, q)
    lda, ldb = q + (q % 2), m + 1
    a = torch.randn(batch, q, lda, dtype=torch.float64, device="cuda", generator=g) * (0.3 / q ** 0.5)
    d = torch.arange(q, device="cuda")
    a[:, d, d] += 1.5
    b = torch.rand(batch, n, ldb, dtype=torch.float64, device="cuda", generator=g)
    x = b.clone()
    level3.trsm_batched_dev(side, uplo, trans, diag, m, n, 0.75, a.data_ptr(), lda, q * lda, x.data_ptr(), ldb, n * ldb, batch,
                            np.float64, stream=torch.cuda.current_stream().cuda_stream)
    t = a[:, :, :q].transpose(1, 2)  # column-major storage
    t = torch.triu(t) if uplo == Uplo.Upper else torch.tril(t)
    if diag == Diag.Unit:
        t = t - torch.diag_embed(torch.diagonal(t, dim1=1, dim2=2)) + torch.eye(q, dtype=t.dtype, device="cuda")
    op = t.transpose(1, 2) if trans == Transpose.Trans else t
    X, B = x[:, :, :m].transpose(1, 2), b[:, :, :m].transpose(1, 2)
    r = (op @ X if side == Side.Left else X @ op) - 0.75 * B
    norm = lambda v: torch.linalg.vector_norm(v, dim=(1, 2))
    err = norm(r) / (norm(op) * norm(X) + 0.75 * norm(B))
    assert float(err.max()) <= 4 * q * 2.0 ** -53
    assert torch.equal(x[:, :, m:], b[:, :, m:])  # padding untouched
    assert rb.device_error()[0] == 0
