"""GPU test of gemv's order of summation where one thread per row fills the GPU:
a NoTrans column-major call of that many rows adds its columns in rblas's order,
so it equals the oracle bit for bit, however many columns it has."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import rblas_b200 as rb
from rblas_b200 import complex2, level2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ROWS = 1183 * 1024 + 1  # the fewest


@pytest.mark.parametrize("dt,n", [("float32", 32), ("float32", 67), ("float64", 33), ("complex64", 32)])
def test_many_rows_keep_rblas_order(dt, n):
    rng = np.random.default_rng(n)
    ndt = np.dtype(dt)

    def rand(k):
        v = rng.standard_normal(k)
        return (v + 1j * rng.standard_normal(k) if ndt.kind == "c" else v).astype(ndt)

    a, x, y = rand(ROWS * n), rand(n), rand(ROWS)
    da, dx, dy = (torch.from_numpy(v).cuda() for v in (a, x, y))
    mod = complex2 if ndt.kind == "c" else level2
    mod.gemv_dev(1, 0, ROWS, n, 0.75, da.data_ptr(), ROWS, dx.data_ptr(), 1, -0.5, dy.data_ptr(), 1, ndt,
                 stream=torch.cuda.current_stream().cuda_stream)
    oracle.gemv(1, 0, ROWS, n, 0.75, a, ROWS, x, 1, -0.5, y, 1)
    assert np.array_equal(dy.cpu().numpy(), y)
    assert rb.device_error()[0] == 0
