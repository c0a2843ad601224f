"""GPU tests of the autotuner's Ozaki tile widths: a width is timed for exactly
the shape buckets that hold a shape whose call reads it, that is, one that does
not run on CTA pairs; and at shapes that read it, either width gives the same
bits, in single calls and in a grouped launch beside pairs."""
from __future__ import annotations

import numpy as np
import pytest

from rblas_b200 import level3
from rblas_b200.serving import Problem, autotune, autotune_load, autotune_reset, grouped_gemm_ozaki
from rblas_b200.types import Layout, Precision

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def on_pairs(m, n):
    if m <= 128:
        return False
    t = lambda x, w: -(-x // w)
    return n <= 128 or 0.85 * t(m, 256) * t(n, 128) <= float(t(m, 128) * t(n, 256))


def test_widths_are_timed_where_they_are_read(tmp_path):
    cache = tmp_path / "tuned.txt"
    try:
        autotune(str(cache))
    finally:
        autotune_reset()
    rows = [tuple(int(x) for x in ln.split()) for ln in cache.read_text().splitlines()[2:]]
    timed = {r[1:4] for r in rows if r[0] == 2}
    read = {(lm, ln) for lm in range(5, 13) for ln in range(5, 11)
            if any(not on_pairs(m, n) for m in range(1 << lm, 2 << lm) for n in range(1 << ln, 2 << ln, 16))}
    assert timed == {(lm, ln, lk) for lm, ln in read for lk in range(5, 13)}


def test_either_width_gives_the_same_bits(tmp_path):
    shapes = [(300, 200, 700), (513, 129, 1025), (100, 700, 300), (640, 1000, 500), (700, 600, 900)]
    assert [on_pairs(m, n) for m, n, _ in shapes] == [False] * 4 + [True]
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    ops = [[torch.randn(s, dtype=torch.float64, device="cuda", generator=g) for s in (m * k, k * n, m * n)]
           for m, n, k in shapes]
    prop = torch.cuda.get_device_properties(0)
    head = f"rblas_b200 grouped autotune v2\ndevice {prop.name.replace(' ', '_')} {prop.multi_processor_count}\n"
    results = []
    try:
        for width in (128, 256):
            cache = tmp_path / f"w{width}.txt"
            cache.write_text(head + "".join(f"2 {lm} {ln} {lk} {width}\n" for lm in range(5, 13) for ln in range(5, 13)
                                            for lk in range(5, 13)))
            autotune_load(str(cache))
            single, group = ([c.clone() for _, _, c in ops] for _ in range(2))
            for (m, n, k), (a, b, _), c in zip(shapes, ops, single):
                level3.gemm_dev(Layout.ColMajor, 0, 0, m, n, k, 1.25, a.data_ptr(), m, b.data_ptr(), k, -0.5, c.data_ptr(), m,
                                np.float64, prec=Precision.Ozaki)
            torch.cuda.synchronize()
            grouped_gemm_ozaki([Problem(np.float64, Layout.ColMajor, 0, 0, m, n, k, 1.25, a.data_ptr(), m, b.data_ptr(), k, -0.5,
                                        c.data_ptr(), m) for (m, n, k), (a, b, _), c in zip(shapes, ops, group)])
            torch.cuda.synchronize()
            results += [single, group]
    finally:
        autotune_reset()
    for r in results[1:]:
        assert all(torch.equal(x.view(torch.int64), y.view(torch.int64)) for x, y in zip(r, results[0]))
