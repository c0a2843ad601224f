"""Performance cases: the calls that programs make of this library, through
its Python entry points, over the sizes they make them at.

A case is a dict of plain values. `listed()` gives the fixed cases, `draw(rng)`
one more of the same ranges, `prepare` the operands a program has in hand,
`run` one pass, `work` the bytes and operations a pass cannot do without, and
`exact` the same outputs in 64 bits by plain torch / numpy.

Families (the `op` of a case):
  host   level3.gemm on numpy slices: rblas's own call, transfers included
  gemm   level3.gemm_dev on device pointers, in any arithmetic form
  cgemm  complex3.gemm_dev
  trsm   level3.trsm_batched_dev, or level3.trsm_dev for one problem
  gemv   level2.gemv_dev
  ger    level2.ger_dev
  vec    the vector work of one Krylov step (axpy, dot, nrm2 through level1)
  batch  one admitted set of a GEMM server: the grouped launches
"""
from __future__ import annotations

import random

import numpy as np
import torch

from rblas_b200 import complex3, level1, level2, level3, serving
from rblas_b200.types import Diag, Layout, Precision, Side, Transpose, Uplo

FORMS = {"plain": Precision.Plain, "ozaki": Precision.Ozaki, "bf16x3": Precision.Bf16x3, "bf16x6": Precision.Bf16x6}
REAL = {"f32": (torch.float32, np.float32), "f64": (torch.float64, np.float64)}
CPLX = {"f32": (torch.complex64, np.complex64), "f64": (torch.complex128, np.complex128)}


def _gemm(name, m, n, k, dt, form, layout="col", ta="n", tb="n", alpha=1.0, beta=0.0, pad=0):
    return {"name": name, "op": "gemm", "m": m, "n": n, "k": k, "dt": dt, "form": form, "layout": layout, "ta": ta, "tb": tb,
            "alpha": alpha, "beta": beta, "pad": pad}


def listed():
    return [
        # The smallest call of a program that moves from rblas: ordinary host
        # slices, the smallest size rblas's own tables quote. Launches, copies
        # and synchronisation are all there is to it.
        {"name": "host_sgemm_256", "op": "host", "m": 256, "n": 256, "k": 256, "dt": "f32", "form": "plain",
         "layout": "row", "ta": "n", "tb": "n", "alpha": 1.0, "beta": 0.0},
        # The drop-in configuration: 1024^3 SGEMM, resident operands.
        _gemm("sgemm_1024", 1024, 1024, 1024, "f32", "plain"),
        # An ordinary SGEMM on a block of a larger array: odd sizes, a leading
        # dimension that is no multiple of 16 bytes, a transposed operand.
        _gemm("sgemm_ragged", 3001, 2187, 2501, "f32", "plain", layout="row", ta="t", alpha=1.5, beta=0.5, pad=3),
        # FP64 products in true FP64 (the drop-in), a rank-2048 update.
        _gemm("dgemm_plain", 4096, 4096, 2048, "f64", "plain", ta="n", tb="t", alpha=-1.0, beta=1.0),
        # The same in the INT8-slice form, at the benchmark's uneven shape.
        _gemm("dgemm_ozaki_uneven", 3000, 5000, 2048, "f64", "ozaki", layout="row", alpha=1.5, beta=-0.5),
        # The largest: an 8192^3 SGEMM at full FP32 accuracy on tensor cores.
        _gemm("sgemm_bf16x6_8192", 8192, 8192, 8192, "f32", "bf16x6", beta=1.0),
        # Tall and skinny (a projection of many rows on few columns).
        _gemm("sgemm_bf16x3_tall", 65536, 128, 8192, "f32", "bf16x3", alpha=1.0, beta=1.0),
        # Complex: conj(A)^T B in the INT8-slice form.
        {"name": "zgemm_ozaki_2048", "op": "cgemm", "m": 2048, "n": 2048, "k": 2048, "dt": "f64", "form": "ozaki", "ta": "c", "tb": "n",
         "beta0": True},
        # Many small triangular systems (block preconditioners).
        {"name": "dtrsm_batched", "op": "trsm", "q": 512, "r": 64, "batch": 1024, "dt": "f64", "side": "l", "uplo": "l", "trans": "n",
         "unit": False},
        # A matrix-vector product with an ordinary rectangular matrix.
        {"name": "dgemv_t", "op": "gemv", "m": 6000, "n": 4000, "dt": "f64", "layout": "col", "trans": "t", "pad": 0},
        # The vector part of one Krylov iteration at rblas's benchmark length.
        {"name": "krylov_1m", "op": "vec", "n": 1 << 20, "dt": "f32"},
        # One admitted set of the serving stream: mixed sizes, both types, all
        # layouts and transposes; large requests in the precision forms.
        {"name": "serve_64", "op": "batch", "count": 64, "lo": 32, "hi": 4096, "set": 5},
    ]


def _logint(rng, lo, hi):
    v = int(round(lo * (hi / lo) ** rng.random()))
    if rng.random() < 0.5:  # half of the sizes round, half as they fall (odd ones among them)
        v = (v + 31) // 32 * 32
    return max(lo, min(hi, v))


def _dims(rng, lo, hi, most):
    while True:
        m, n, k = (_logint(rng, lo, hi) for _ in range(3))
        if 2.0 * m * n * k <= most:
            return m, n, k


def draw(rng: random.Random):
    op = rng.choice(["host", "splain", "dplain", "ozaki", "bf16", "tall", "cgemm", "trsm", "trsm1", "gemv", "ger", "vec", "batch"])
    lay, ta, tb = rng.choice(["row", "col"]), rng.choice("nt"), rng.choice("nt")
    alpha, beta = rng.choice([1.0, 1.5, -1.0]), rng.choice([0.0, 1.0, -0.5])
    dt = rng.choice(["f32", "f64"])
    if op == "host":
        m, n, k = _dims(rng, 32, 1024, 2.2e9)
        return {"op": "host", "m": m, "n": n, "k": k, "dt": dt, "form": "plain", "layout": lay, "ta": ta, "tb": tb, "alpha": alpha, "beta": beta}
    if op in ("splain", "dplain", "ozaki", "bf16", "tall"):
        if op == "tall":
            dt, form = "f32", rng.choice(["bf16x3", "bf16x6", "plain"])
            m, n, k = _logint(rng, 4096, 65536), _logint(rng, 16, 256), _logint(rng, 512, 8192)
            ta = rng.choice("nnt")
        else:
            dt, form, lo, hi, most = {
                "splain": ("f32", "plain", 64, 4096, 1.4e11), "dplain": ("f64", "plain", 64, 4096, 7.0e10),
                "ozaki": ("f64", "ozaki", 256, 8192, 2.8e11), "bf16": ("f32", rng.choice(["bf16x3", "bf16x6"]), 256, 8192, 1.1e12)}[op]
            m, n, k = _dims(rng, lo, hi, most)
        c = _gemm("", m, n, k, dt, form, layout=lay, ta=ta, tb=tb, alpha=alpha, beta=beta, pad=rng.choice([0, 0, 0, 4, 3]))
        del c["name"]
        return c
    if op == "cgemm":
        m, n, k = _dims(rng, 128, 2048, 1.72e10)
        return {"op": "cgemm", "m": m, "n": n, "k": k, "dt": dt, "form": rng.choice(["plain", "ozaki"] if dt == "f64" else ["plain", "bf16x3", "bf16x6"]),
                "ta": rng.choice("ntc"), "tb": rng.choice("ntc"), "beta0": rng.random() < 0.5}
    if op == "trsm":
        return {"op": "trsm", "q": _logint(rng, 32, 512), "r": _logint(rng, 8, 64), "batch": _logint(rng, 64, 1024), "dt": dt, "side": rng.choice("lr"),
                "uplo": rng.choice("lu"), "trans": rng.choice("nt"), "unit": rng.random() < 0.3}
    if op == "trsm1":
        return {"op": "trsm", "q": _logint(rng, 512, 4096), "r": _logint(rng, 64, 4096), "batch": 1, "dt": "f64", "side": rng.choice("lr"),
                "uplo": rng.choice("lu"), "trans": rng.choice("nt"), "unit": False}
    if op == "gemv":
        return {"op": "gemv", "m": _logint(rng, 256, 16384), "n": _logint(rng, 256, 16384), "dt": dt, "layout": lay, "trans": ta, "pad": rng.choice([0, 0, 3])}
    if op == "ger":
        return {"op": "ger", "m": _logint(rng, 256, 16384), "n": _logint(rng, 256, 16384), "dt": dt, "layout": lay, "pad": rng.choice([0, 0, 3])}
    if op == "vec":
        return {"op": "vec", "n": _logint(rng, 1024, 1 << 26), "dt": dt}
    return {"op": "batch", "count": _logint(rng, 16, 192), "lo": 32, "hi": rng.choice([1024, 2048, 4096]), "set": rng.randrange(1 << 20)}


# ---- operands --------------------------------------------------------------------

_T = {"n": Transpose.NoTrans, "t": Transpose.Trans, "c": Transpose.ConjTrans}
_L = {"row": Layout.RowMajor, "col": Layout.ColMajor}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _uni(count, dtype, g):
    """Uniform on [-1, 1)."""
    return torch.rand(count, dtype=dtype, device="cuda", generator=g).mul_(2).sub_(1)


def _stored(rows, cols, layout, pad):
    """(leading dimension, elements) of a rows x cols matrix."""
    lead = (cols if layout == "row" else rows) + pad
    return lead, lead * (rows if layout == "row" else cols)


def _view(flat, rows, cols, lead, layout):
    return flat.as_strided((rows, cols), (lead, 1) if layout == "row" else (1, lead), flat.storage_offset())


def _shape(case, which):
    m, n, k = case["m"], case["n"], case["k"]
    if which == "a":
        return (m, k) if case["ta"] == "n" else (k, m)
    if which == "b":
        return (k, n) if case["tb"] == "n" else (n, k)
    return m, n


def _op(x, t):
    return x if t == "n" else x.T if t == "t" else x.T.conj()


def _gemm_state(case, seed):
    tdt, g, pad = REAL[case["dt"]][0], _gen(seed), case.get("pad", 0)
    s = {}
    for w in "abc":
        lead, count = _stored(*_shape(case, w), case["layout"], pad)
        s[w], s["ld" + w] = _uni(count, tdt, g), lead
    return s


def _cgemm_state(case, seed):
    tdt, g = CPLX[case["dt"]][0], _gen(seed)
    s = {}
    for w in "abc":
        lead, count = _stored(*_shape(case, w), "col", 0)
        s[w], s["ld" + w] = torch.randn(count, dtype=tdt, device="cuda", generator=g), lead
    return s


def _host_state(case, seed):
    rng = np.random.default_rng(int(seed) + 101)
    s = {}
    for w in "abc":
        lead, count = _stored(*_shape(case, w), case["layout"], 0)
        s[w], s["ld" + w] = rng.uniform(-1, 1, count).astype(REAL[case["dt"]][1]), lead
    return s


def _trsm_state(case, seed):
    """Triangular factors with a unit-size diagonal and small off-diagonal
    entries, so that repeated solves keep their size."""
    g, tdt = _gen(seed), REAL[case["dt"]][0]
    q, r, batch = case["q"], case["r"], case["batch"]
    a = torch.randn(batch, q, q, dtype=tdt, device="cuda", generator=g) * (0.1 / q ** 0.5)
    sign = torch.rand(batch, q, dtype=tdt, device="cuda", generator=g).sub_(0.5).sign_()
    a.diagonal(dim1=1, dim2=2).add_(sign)
    return {"a": a.view(-1), "b": _uni(batch * q * r, tdt, g)}


def _gemv_state(case, seed):
    g, tdt = _gen(seed), REAL[case["dt"]][0]
    lead, count = _stored(case["m"], case["n"], case["layout"], case["pad"])
    short = case["op"] == "ger" or case["trans"] == "n"
    lx, ly = (case["m"], case["n"]) if case["op"] == "ger" else (case["n"], case["m"]) if short else (case["m"], case["n"])
    return {"a": torch.randn(count, dtype=tdt, device="cuda", generator=g), "lda": lead,
            "x": torch.randn(lx, dtype=tdt, device="cuda", generator=g), "y": torch.randn(ly, dtype=tdt, device="cuda", generator=g)}


def _vec_state(case, seed):
    g, tdt = _gen(seed), REAL[case["dt"]][0]
    v = [torch.randn(case["n"], dtype=tdt, device="cuda", generator=g) for _ in range(4)]
    return {"x": v[0], "r": v[1], "p": v[2], "q": v[3], "out": torch.zeros(2, dtype=tdt, device="cuda")}


def _requests(case):
    """The set's requests: shapes, types, layouts and scalars (no data)."""
    rng = np.random.default_rng(case["set"])
    reqs, used = [], [0, 0]
    for _ in range(case["count"]):
        m, n, k = (int(round(float(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"])))))) for _ in range(3))
        d, row, ta, tb = (int(v) for v in rng.integers(0, 2, 4))
        q = {"m": m, "n": n, "k": k, "d": d, "layout": "row" if row else "col", "ta": "nt"[ta], "tb": "nt"[tb],
             "alpha": float(np.float32(rng.uniform(-2, 2))), "beta": float(np.float32(rng.uniform(-1, 1)))}
        for w in "abc":  # leading dimensions and offsets on 16 bytes, as an allocator gives them
            rows, cols = _shape(q, w)
            lead = ((cols if row else rows) + 3) // 4 * 4
            q["ld" + w], q["len" + w] = lead, lead * (rows if row else cols)
        most = max(q["lena"], q["lenb"])
        q["offa"], q["offb"] = (int(rng.integers(0, (1 << 25) - most)) // 4 * 4 for _ in range(2))
        q["offc"] = used[d]
        used[d] += (q["lenc"] + 3) // 4 * 4
        reqs.append(q)
    return reqs, used


def _batch_state(case, seed):
    reqs, used = _requests(case)
    g = _gen(seed)
    pools = [torch.randn(1 << 25, dtype=t, device="cuda", generator=g) for t in (torch.float32, torch.float64)]
    c = [torch.randn(max(4, used[d]), dtype=t, device="cuda", generator=g) for d, t in enumerate((torch.float32, torch.float64))]
    plain, x6, oz = [], [], []
    for q in reqs:
        el = 8 if q["d"] else 4
        p = serving.Problem(np.float64 if q["d"] else np.float32, _L[q["layout"]], _T[q["ta"]], _T[q["tb"]], q["m"], q["n"], q["k"], q["alpha"],
                            pools[q["d"]].data_ptr() + el * q["offa"], q["lda"], pools[q["d"]].data_ptr() + el * q["offb"], q["ldb"], q["beta"],
                            c[q["d"]].data_ptr() + el * q["offc"], q["ldc"])
        flop = 2.0 * q["m"] * q["n"] * q["k"]
        # the serving configuration's thresholds
        (oz if q["d"] and flop >= 1e9 else x6 if not q["d"] and flop >= 2e8 else plain).append(p)
    return {"pools": pools, "c": c, "plain": plain, "x6": x6, "oz": oz}


def prepare(case, seed):
    make = {"gemm": _gemm_state, "cgemm": _cgemm_state, "host": _host_state, "trsm": _trsm_state, "gemv": _gemv_state, "ger": _gemv_state,
            "vec": _vec_state, "batch": _batch_state}[case["op"]]
    s = make(case, seed)
    s["case"] = case
    return s


# ---- one pass --------------------------------------------------------------------

ALPHA_C, BETA_C = complex(1.0, 0.5), complex(0.25, -0.5)


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "host":
        level3.gemm(_L[case["layout"]], _T[case["ta"]], _T[case["tb"]], case["m"], case["n"], case["k"], case["alpha"], s["a"], s["lda"], s["b"], s["ldb"],
                    case["beta"], s["c"], s["ldc"], prec=FORMS[case["form"]])
        return s["c"]
    st = torch.cuda.current_stream().cuda_stream
    if op == "gemm":
        level3.gemm_dev(_L[case["layout"]], _T[case["ta"]], _T[case["tb"]], case["m"], case["n"], case["k"], case["alpha"], s["a"].data_ptr(), s["lda"],
                        s["b"].data_ptr(), s["ldb"], case["beta"], s["c"].data_ptr(), s["ldc"], REAL[case["dt"]][1], prec=FORMS[case["form"]], stream=st)
        return s["c"]
    if op == "cgemm":
        complex3.gemm_dev(_T[case["ta"]], _T[case["tb"]], case["m"], case["n"], case["k"], ALPHA_C, s["a"].data_ptr(), s["lda"], s["b"].data_ptr(), s["ldb"],
                          0.0 if case["beta0"] else BETA_C, s["c"].data_ptr(), s["ldc"], CPLX[case["dt"]][1], prec=FORMS[case["form"]], stream=st)
        return s["c"]
    if op == "trsm":
        q, r = case["q"], case["r"]
        m, n = (q, r) if case["side"] == "l" else (r, q)
        args = (Side.Left if case["side"] == "l" else Side.Right, Uplo.Lower if case["uplo"] == "l" else Uplo.Upper, _T[case["trans"]],
                Diag.Unit if case["unit"] else Diag.NonUnit, m, n, 1.0)
        if case["batch"] == 1:
            level3.trsm_dev(*args, s["a"].data_ptr(), q, s["b"].data_ptr(), m, stream=st)
        else:
            level3.trsm_batched_dev(*args, s["a"].data_ptr(), q, q * q, s["b"].data_ptr(), m, m * n, case["batch"], REAL[case["dt"]][1], stream=st)
        return s["b"]
    if op == "gemv":
        level2.gemv_dev(_L[case["layout"]], _T[case["trans"]], case["m"], case["n"], 1.25, s["a"].data_ptr(), s["lda"], s["x"].data_ptr(), 1, 0.5,
                        s["y"].data_ptr(), 1, REAL[case["dt"]][1], stream=st)
        return s["y"]
    if op == "ger":
        level2.ger_dev(_L[case["layout"]], case["m"], case["n"], 1.25, s["x"].data_ptr(), 1, s["y"].data_ptr(), 1, s["a"].data_ptr(), s["lda"],
                       REAL[case["dt"]][1], stream=st)
        return s["a"]
    if op == "vec":
        n, dt, el = case["n"], REAL[case["dt"]][1], s["out"].element_size()
        level1.axpy_dev(n, 0.125, s["p"].data_ptr(), 1, s["x"].data_ptr(), 1, dt, stream=st)
        level1.axpy_dev(n, -0.125, s["q"].data_ptr(), 1, s["r"].data_ptr(), 1, dt, stream=st)
        level1.dot_dev(n, s["r"].data_ptr(), 1, s["p"].data_ptr(), 1, s["out"].data_ptr(), dt, stream=st)
        level1.nrm2_dev(n, s["r"].data_ptr(), 1, s["out"].data_ptr() + el, dt, stream=st)
        return {"x": s["x"], "r": s["r"], "out": s["out"]}
    if s["oz"]:
        serving.grouped_gemm_ozaki(s["oz"], stream=st)
    if s["x6"]:
        serving.grouped_gemm_bf16(s["x6"], Precision.Bf16x6, stream=st)
    if s["plain"]:
        serving.grouped_gemm(s["plain"], stream=st)
    return s["c"]


# ---- work and exact results ----------------------------------------------------------

def work(case):
    op = case["op"]
    el = 8 if case.get("dt") == "f64" else 4
    if op in ("gemm", "host", "cgemm"):
        m, n, k = case["m"], case["n"], case["k"]
        reads_c = (not case["beta0"]) if op == "cgemm" else case["beta"] != 0.0
        w = 2 if op == "cgemm" else 1
        return {"bytes": w * el * (m * k + k * n + m * n * (2 if reads_c else 1)), "flops": (8.0 if op == "cgemm" else 2.0) * m * n * k}
    if op == "trsm":
        q, r, b = case["q"], case["r"], case["batch"]
        return {"bytes": el * b * (q * (q + 1) // 2 + 2 * q * r), "flops": float(b) * q * q * r}
    if op == "gemv":
        m, n = case["m"], case["n"]
        ly = m if case["trans"] == "n" else n
        return {"bytes": el * (m * n + m + n + ly), "flops": 2.0 * m * n}
    if op == "ger":
        m, n = case["m"], case["n"]
        return {"bytes": el * (2 * m * n + m + n), "flops": 2.0 * m * n}
    if op == "vec":  # p, q and r's and x's old values in, r and x out (the reductions' operands are then at hand)
        return {"bytes": el * 6 * case["n"], "flops": 8.0 * case["n"]}
    total, flops = 0, 0.0
    for q in _requests(case)[0]:
        total += (8 if q["d"] else 4) * (q["m"] * q["k"] + q["k"] * q["n"] + 2 * q["m"] * q["n"])
        flops += 2.0 * q["m"] * q["n"] * q["k"]
    return {"bytes": total, "flops": flops}


def _exact_gemm(case, a, lda, b, ldb, c, ldc, alpha, beta, layout):
    """alpha*op(A)*op(B) + beta*C in 64 bits, as C's flat buffer (its padding as it was)."""
    wide = torch.complex128 if c.is_complex() else torch.float64
    out = c.to(wide)
    oa = _op(_view(a, *_shape(case, "a"), lda, layout).to(wide), case["ta"])
    ob = _op(_view(b, *_shape(case, "b"), ldb, layout).to(wide), case["tb"])
    cv = _view(out, *_shape(case, "c"), ldc, layout)
    cv.copy_(alpha * (oa @ ob) + (beta * cv if beta != 0 else 0))
    return out


def exact(case, seed):
    s = prepare(case, seed)
    op = case["op"]
    if op == "host":
        t = {w: torch.from_numpy(s[w]) for w in "abc"}
        return _exact_gemm(case, t["a"], s["lda"], t["b"], s["ldb"], t["c"], s["ldc"], case["alpha"], case["beta"], case["layout"]).numpy()
    if op == "gemm":
        return _exact_gemm(case, s["a"], s["lda"], s["b"], s["ldb"], s["c"], s["ldc"], case["alpha"], case["beta"], case["layout"])
    if op == "cgemm":
        return _exact_gemm(case, s["a"], s["lda"], s["b"], s["ldb"], s["c"], s["ldc"], ALPHA_C, 0.0 if case["beta0"] else BETA_C, "col")
    if op == "trsm":
        q, r, batch = case["q"], case["r"], case["batch"]
        m, n = (q, r) if case["side"] == "l" else (r, q)
        out = torch.empty(batch, n, m, dtype=torch.float64, device="cuda")
        for i in range(0, batch, 128):  # a column-major block is the transpose of the row-major view
            a = s["a"].view(batch, q, q)[i:i + 128].transpose(1, 2).double()
            b = s["b"].view(batch, n, m)[i:i + 128].transpose(1, 2).double()
            upper = case["uplo"] == "u"
            if case["trans"] == "t":
                a, upper = a.transpose(1, 2), not upper
            x = torch.linalg.solve_triangular(a, b, upper=upper, left=case["side"] == "l", unitriangular=case["unit"])
            out[i:i + 128] = x.transpose(1, 2)
        return out.view(-1)
    if op in ("gemv", "ger"):
        a = s["a"].double()
        v = _view(a, case["m"], case["n"], s["lda"], case["layout"])
        if op == "ger":
            v.add_(torch.outer(1.25 * s["x"].double(), s["y"].double()))
            return a
        return 1.25 * (_op(v, case["trans"]) @ s["x"].double()) + 0.5 * s["y"].double()
    if op == "vec":
        x = s["x"].double() + 0.125 * s["p"].double()
        r = s["r"].double() - 0.125 * s["q"].double()
        return {"x": x, "r": r, "out": torch.stack([torch.dot(r, s["p"].double()), torch.linalg.vector_norm(r)])}
    c = [t.double() for t in s["c"]]
    for q in _requests(case)[0]:
        d = q["d"]
        a, b = (s["pools"][d][q["off" + w]:q["off" + w] + q["len" + w]] for w in "ab")
        at = slice(q["offc"], q["offc"] + q["lenc"])
        c[d][at] = _exact_gemm(q, a, q["lda"], b, q["ldb"], s["c"][d][at], q["ldc"], q["alpha"], q["beta"], q["layout"])
    return c
