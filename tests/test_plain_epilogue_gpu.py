"""GPU test of the plain GEMM's epilogue where some of a tile's warps have no
rows or columns of C, with and without C0: within 4 k u of the oracle, NaN in C
when beta is 0 leaves no trace, and what lies between C's columns is untouched."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import rblas_b200 as rb
from rblas_b200 import level3

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("beta", [0.0, 1.0, -0.5])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 10), (64, 16), (65, 17), (63, 65), (130, 49), (1, 200), (200, 1)])
def test_tiles_with_idle_warps(dt, beta, m, n):
    k, ldc = 2400, m + 3  # long enough a K to run on the 128-wide tiles
    rng = np.random.default_rng(m * 7 + n)
    a, b, c = (rng.uniform(-1, 1, s).astype(dt) for s in (m * k, k * n, ldc * n))
    if beta == 0.0:
        c.reshape(n, ldc)[:, :m] = np.nan
    da, db, dc = (torch.from_numpy(v).cuda() for v in (a, b, c))
    level3.gemm_dev(1, 0, 0, m, n, k, 1.5, da.data_ptr(), m, db.data_ptr(), k, beta, dc.data_ptr(), ldc, np.dtype(dt),
                    stream=torch.cuda.current_stream().cuda_stream)
    ref = c.copy()
    oracle.gemm(1, 0, 0, m, n, k, 1.5, a, m, b, k, beta, ref, ldc)
    got, want, was = (v.reshape(n, ldc) for v in (dc.cpu().numpy(), ref, c))
    assert np.array_equal(got[:, m:], was[:, m:])
    c0 = 0.0 if beta == 0.0 else abs(beta) * np.linalg.norm(was[:, :m].astype(np.float64))
    den = 1.5 * np.linalg.norm(a.astype(np.float64)) * np.linalg.norm(b.astype(np.float64)) + c0
    u = 2.0 ** -24 if dt == "float32" else 2.0 ** -53
    assert np.linalg.norm(got[:, :m].astype(np.float64) - want[:, :m]) <= 4 * k * u * den
    assert rb.device_error()[0] == 0
