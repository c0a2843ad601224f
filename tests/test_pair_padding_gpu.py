"""GPU test of the CTA-pair kernels on shapes that run on them (the CPU test
test_pair_routes_cpu.py holds the lists below to the dispatch rules), with C's
leading dimension above m: each result equals that of another of the library's
kernels bit for bit, and what lies between C's columns keeps its bits.

Ozaki: whole tiles, a split tail (several K parts of each group of diagonals),
both with one K column and with a K of two INT32 chunks; exponents outside the
moderate range, zero rows and columns, infinities and NaNs; every slice count;
one call and the grouped launch, against the allocation-free entry point.
BF16 split: one, several and a short last accumulation unit, against the
grouped launch. The tall form: against the same matrix stored transposed."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import rblas_b200 as rb
from rblas_b200 import _lib, level3, serving
from rblas_b200.types import Layout, Precision

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

PAD = 5
OZ_WHOLE = [(513, 257, 1), (256, 128, 1), (520, 260, 200), (1025, 1030, 520), (257, 128, 20000)]
OZ_TAIL = [(300, 300, 3000), (513, 257, 1000), (256, 129, 1000)]
OZ_SLICES = (300, 300, 8000)  # a tail at every slice count
BF16 = [(2047, 2177, 481), (2048, 2304, 129), (1921, 2303, 193), (2047, 2177, 1), (4097, 4609, 97)]
TALL = [(260, 129, 192), (40004, 128, 129), (20000, 256, 321), (512, 3, 65)]


def randn(count, dtype, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(count, dtype=dtype, device="cuda", generator=g)


def same(x, y):
    """Bit for bit, NaNs counting as equal."""
    nx, ny = torch.isnan(x), torch.isnan(y)
    it = torch.int64 if x.dtype == torch.float64 else torch.int32
    return torch.equal(nx, ny) and torch.equal(x.view(it).masked_fill(nx, 0), y.view(it).masked_fill(ny, 0))


def padding_kept(c, c0, m, n):
    return same(c.view(n, m + PAD)[:, m:].contiguous(), c0.view(n, m + PAD)[:, m:].contiguous())


def ozaki(m, n, k, a, b, c0, alpha, beta):
    """The call, the grouped launch and the allocation-free entry point."""
    ldc, st = m + PAD, torch.cuda.current_stream().cuda_stream
    call, group, other = c0.clone(), c0.clone(), c0.clone()
    level3.gemm_dev(Layout.ColMajor, 0, 0, m, n, k, alpha, a.data_ptr(), m, b.data_ptr(), k, beta, call.data_ptr(), ldc,
                    np.float64, prec=Precision.Ozaki, stream=st)
    serving.grouped_gemm_ozaki([serving.Problem(np.float64, Layout.ColMajor, 0, 0, m, n, k, alpha, a.data_ptr(), m,
                                                b.data_ptr(), k, beta, group.data_ptr(), ldc)], stream=st)
    err = _lib.RbError()
    s = _lib.load().rb_dgemm_ozaki_noalloc(1, 0, 0, m, n, k, alpha, C.c_void_p(a.data_ptr()), m, C.c_void_p(b.data_ptr()),
                                           k, beta, C.c_void_p(other.data_ptr()), ldc, C.c_void_p(st) if st else None,
                                           C.byref(err))
    _lib.check(s, err)
    for c in (call, group, other):
        assert padding_kept(c, c0, m, n), (m, n, k)
    assert same(call, other) and same(group, other), (m, n, k)
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0


def ozaki_operands(m, n, k):
    return [randn(s, torch.float64, 3 * m + n + k + i) for i, s in enumerate((m * k, k * n, (m + PAD) * n))]


@pytest.mark.parametrize("m,n,k", OZ_WHOLE + OZ_TAIL)
@pytest.mark.parametrize("beta", [0.0, 1.0, -0.5])
def test_ozaki(m, n, k, beta):
    a, b, c0 = ozaki_operands(m, n, k)
    ozaki(m, n, k, a, b, c0, 1.5, beta)


@pytest.mark.parametrize("slices", range(2, 13))
def test_ozaki_slice_counts(slices):
    lib = _lib.load()
    keep = lib.rb_get_ozaki_slices()
    m, n, k = OZ_SLICES
    a, b, c0 = ozaki_operands(m, n, k)
    try:
        assert lib.rb_set_ozaki_slices(slices) == 0
        ozaki(m, n, k, a, b, c0, -0.75, 1.0)
    finally:
        lib.rb_set_ozaki_slices(keep)


@pytest.mark.parametrize("m,n,k", [OZ_WHOLE[2], OZ_TAIL[0], OZ_TAIL[1]])
@pytest.mark.parametrize("alpha", [1.0, 2.0 ** 400, float("inf")])
def test_ozaki_specials(m, n, k, alpha):
    a, b, c0 = ozaki_operands(m, n, k)
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
    ozaki(m, n, k, a, b, c0, alpha, 1.0)


@pytest.mark.parametrize("form", [Precision.Bf16x3, Precision.Bf16x6])
@pytest.mark.parametrize("m,n,k", BF16)
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_bf16_pairs(form, m, n, k, beta):
    ldc, st = m + PAD, torch.cuda.current_stream().cuda_stream
    # A^T: rows of A are not contiguous, so the tall form does not take it
    a, b, c0 = (randn(s, torch.float32, m + n + k + i) for i, s in enumerate((m * k, k * n, ldc * n)))
    for special in (False, True):
        if special:
            a[(m * k) // 2], b[(k * n) // 3] = float("inf"), float("nan")
        call, group = c0.clone(), c0.clone()
        level3.gemm_dev(Layout.ColMajor, 1, 0, m, n, k, 1.5, a.data_ptr(), k, b.data_ptr(), k, beta, call.data_ptr(), ldc,
                        np.float32, prec=form, stream=st)
        serving.grouped_gemm_bf16([serving.Problem(np.float32, Layout.ColMajor, 1, 0, m, n, k, 1.5, a.data_ptr(), k,
                                                   b.data_ptr(), k, beta, group.data_ptr(), ldc)], form, stream=st)
        assert same(call, group)
        assert padding_kept(call, c0, m, n)
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0


@pytest.mark.parametrize("form", [Precision.Bf16x3, Precision.Bf16x6])
@pytest.mark.parametrize("m,n,k", TALL)
def test_tall_pairs(form, m, n, k):
    ldc, st = m + PAD, torch.cuda.current_stream().cuda_stream
    a, b, c0 = (randn(s, torch.float32, m + n + k + i) for i, s in enumerate((m * k, k * n, ldc * n)))
    at = a.view(k, m).t().contiguous().view(-1)
    tall, two_pass = c0.clone(), c0.clone()
    level3.gemm_dev(Layout.ColMajor, 0, 0, m, n, k, 1.25, a.data_ptr(), m, b.data_ptr(), k, -0.5, tall.data_ptr(), ldc,
                    np.float32, prec=form, stream=st)
    level3.gemm_dev(Layout.ColMajor, 1, 0, m, n, k, 1.25, at.data_ptr(), k, b.data_ptr(), k, -0.5, two_pass.data_ptr(), ldc,
                    np.float32, prec=form, stream=st)
    assert same(tall, two_pass)
    assert padding_kept(tall, c0, m, n)
    torch.cuda.synchronize()
    assert rb.device_error()[0] == 0
