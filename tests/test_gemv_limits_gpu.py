"""GPU test of gemv at the largest row and column counts that its 32-bit indexes
take: every element of A is read once and none past its end is (A of ones, so a
sum is the count; the ranges' sums are whole numbers below 2^24, and adding at
most 1184 of them rounds by 2^-24 each, less than one range's share)."""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import level2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TOP = 2 ** 31 - 1


@pytest.mark.parametrize("count", [TOP, TOP - 5, TOP - 1000])
@pytest.mark.parametrize("m_long", [True, False])
@pytest.mark.parametrize("trans", [0, 1])
def test_largest_counts(count, m_long, trans):
    m, n = (count, 1) if m_long else (1, count)
    summed = n if trans == 0 else m
    # past A's end: NaN, which a read there would leave in a sum
    a = torch.ones(count + 4096, dtype=torch.float32, device="cuda")
    a[count:] = float("nan")
    x = torch.ones(1, dtype=torch.float32, device="cuda")  # incx 0
    y = torch.zeros(m if trans == 0 else n, dtype=torch.float32, device="cuda")
    level2.gemv_dev(1, trans, m, n, 1.0, a.data_ptr(), m, x.data_ptr(), 0, 0.0, y.data_ptr(), 1, np.float32,
                    stream=torch.cuda.current_stream().cuda_stream)
    if summed == 1:
        assert float(y.min()) == 1.0 and float(y.max()) == 1.0
    else:
        assert abs(float(y[0]) / count - 1) <= 1184 * 2.0 ** -24
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
