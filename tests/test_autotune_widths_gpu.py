"""GPU test of the autotuner's Ozaki tile widths: a width is timed for exactly
the shape buckets that hold a shape whose call reads it, that is, one that does
not run on CTA pairs."""
from __future__ import annotations

import pytest

from rblas_b200.serving import autotune, autotune_reset

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


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
