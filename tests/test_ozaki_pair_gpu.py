"""GPU test of the Ozaki GEMM on CTA pairs (256 x 128 tiles, four diagonals at
a time, FP64 sums in registers): at shapes ragged against its tiles, with
whole tiles, a split tail (groups and K parts) and every slice count, the
result equals the allocation-free entry point's (128 x 256 tiles, two
diagonals at a time through C) bit for bit: the same terms are folded in the
same order. Rows, columns and alpha outside the moderate exponents, zero rows
and columns, infinities and NaNs take the general scaling; equal there too.
The allocation-free entry point is checked against the oracle in
test_zz_no_alloc.py.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import _lib, level3
from rblas_b200.types import Layout, Precision, Transpose

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def both(m, n, k, a, b, c0, alpha, beta):
    st = torch.cuda.current_stream().cuda_stream
    c1, c2 = c0.clone(), c0.clone()
    level3.gemm_dev(Layout.ColMajor, Transpose.NoTrans, Transpose.NoTrans, m, n, k, alpha, a.data_ptr(), m, b.data_ptr(), k, beta,
                    c1.data_ptr(), m, np.float64, prec=Precision.Ozaki, stream=st)
    err = _lib.RbError()
    s = _lib.load().rb_dgemm_ozaki_noalloc(1, 0, 0, m, n, k, alpha, C.c_void_p(a.data_ptr()), m, C.c_void_p(b.data_ptr()), k, beta,
                                           C.c_void_p(c2.data_ptr()), m, C.c_void_p(st) if st else None, C.byref(err))
    _lib.check(s, err)
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
    return c1, c2


def operands(m, n, k, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [torch.randn(s, dtype=torch.float64, device="cuda", generator=g) for s in (m * k, k * n, m * n)]


@pytest.mark.parametrize("m,n,k,beta", [
    (256, 128, 128, 0.0), (257, 129, 1, 1.0), (511, 127, 127, -0.5), (513, 257, 129, 1.0), (300, 300, 3000, 0.5),
    (1025, 1030, 520, -0.5), (1800, 1700, 300, 1.0)])
def test_pair_tiles(m, n, k, beta):
    a, b, c0 = operands(m, n, k, m + k)
    c1, c2 = both(m, n, k, a, b, c0, 1.5, beta)
    assert torch.equal(c1.view(torch.int64), c2.view(torch.int64))


@pytest.mark.parametrize("slices", range(2, 13))
def test_slice_counts(slices):
    lib = _lib.load()
    keep = lib.rb_get_ozaki_slices()
    try:
        assert lib.rb_set_ozaki_slices(slices) == 0
        for m, n, k in ((520, 260, 400), (300, 140, 2000)):
            a, b, c0 = operands(m, n, k, slices)
            c1, c2 = both(m, n, k, a, b, c0, -0.75, 1.0)
            assert torch.equal(c1.view(torch.int64), c2.view(torch.int64)), (m, n, k)
    finally:
        lib.rb_set_ozaki_slices(keep)


@pytest.mark.parametrize("alpha", [1.0, 2.0 ** 400, float("inf")])
def test_exponents_and_specials(alpha):
    for m, n, k in ((520, 260, 200), (300, 140, 2000)):
        a, b, c0 = operands(m, n, k, 5)
        av, bv = a.view(k, m), b.view(n, k)  # column-major: [column][row]
        av[:, 3] *= 2.0 ** 1000
        av[:, 130] *= 2.0 ** -1000
        av[:, 260] *= 2.0 ** 300
        av[:, 7] = 0
        bv[5] *= 2.0 ** -1030
        bv[130] *= 2.0 ** 500
        bv[9] = 0
        av[0, 11] = float("inf")
        bv[17, 1] = float("nan")
        c1, c2 = both(m, n, k, a, b, c0, alpha, 1.0)
        assert torch.equal(torch.isnan(c1), torch.isnan(c2))
        assert torch.equal(c1.nan_to_num(0.0, 1.0, 2.0), c2.nan_to_num(0.0, 1.0, 2.0))
        assert torch.equal(torch.isposinf(c1), torch.isposinf(c2))
