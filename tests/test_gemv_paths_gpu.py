"""GPU test of gemv's paths at the edges of their tiles: few and many columns,
short and long columns, ranges, operands on and off 16 bytes, strided x and y,
every type, against the 64-bit product within 4 K u sum |a||x| (K terms, one
rounding each, plus the final steps)."""
from __future__ import annotations

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import complex2, level2
from rblas_b200.types import Layout, Transpose

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 1), (63, 31), (64, 32), (65, 33), (1000, 31), (129, 700), (7, 5001), (5001, 7), (2049, 1025), (1024, 4736), (1021, 4739),
          (9000, 260)]


@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
@pytest.mark.parametrize("trans", [Transpose.NoTrans, Transpose.Trans, Transpose.ConjTrans])
@pytest.mark.parametrize("pad,off,inc", [(0, 0, 1), (1, 0, 1), (0, 1, 1), (2, 0, 3)])
def test_gemv_paths(dt, trans, pad, off, inc):
    tdt, ndt = getattr(torch, dt), np.dtype(dt)
    wide = torch.complex128 if tdt.is_complex else torch.float64
    u = 2.0 ** -24 if dt in ("float32", "complex64") else 2.0 ** -53
    g = torch.Generator(device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    for m, n in SHAPES:
        g.manual_seed(m * 31 + n)
        ld = m + pad
        a = torch.randn(off + ld * n, dtype=tdt, device="cuda", generator=g)[off:]
        k, ly = (n, m) if trans == Transpose.NoTrans else (m, n)
        x = torch.randn(k * inc, dtype=tdt, device="cuda", generator=g)
        y = torch.randn(ly * inc, dtype=tdt, device="cuda", generator=g)
        y0 = y.clone()
        mod = complex2 if tdt.is_complex else level2
        lay = () if tdt.is_complex and "layout" not in mod.gemv_dev.__code__.co_varnames else (Layout.ColMajor,)
        mod.gemv_dev(*lay, trans, m, n, 1.25, a.data_ptr(), ld, x.data_ptr(), inc, 0.5, y.data_ptr(), inc, ndt, stream=st)
        op = a.as_strided((m, n), (1, ld), a.storage_offset()).to(wide)
        op = op if trans == Transpose.NoTrans else op.T if trans == Transpose.Trans else op.T.conj()
        xs, ys = x[::inc].to(wide), y0[::inc].to(wide)
        exact = 1.25 * (op @ xs) + 0.5 * ys
        size = 1.25 * (op.abs() @ xs.abs()) + 0.5 * ys.abs()
        off_by = (y[::inc].to(wide) - exact).abs()
        assert bool((off_by <= 4 * (k + 4) * u * size).all()), (m, n)
        if inc > 1:  # the elements between the strides are untouched
            assert torch.equal(y.view(-1, inc)[:, 1:], y0.view(-1, inc)[:, 1:])
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
