"""The calls whose speed this library is judged by, through its public entry points.

Every case is a dict of plain values with a "kind":

  red      a value-returning reduction of device vectors (reproBLAS_r{d,s,z,c}{sum,dot,nrm2})
  gemv     reproBLAS_r{d,s,z,c}gemv, row-major, device operands, y written in place (beta 0)
  gemm     reproBLAS_r{d,s,z,c}gemm, row-major, device operands, C written in place (beta 0)
  int8     rb_dgemm_int8, the int8-sliced dgemm on the tensor cores
  batch    rb_batch_plan_run: ragged dot products and small dgemms in one launch

listed() names the ones that are followed, draw() gives others of the same ranges. prepare()
makes the device operands (and the batch plan), run() makes the one call and returns its
outputs, exact() is the same value from plain torch in 64 bits.
"""
import ctypes
import math

import torch

import reproblas_b200 as rb

_REAL = {"d": torch.float64, "s": torch.float32, "z": torch.float64, "c": torch.float32}


def listed():
    return [
        # a scalar product inside an iterative solver's small system: latency only
        {"name": "ddot_4k", "kind": "red", "type": "d", "op": "dot", "fold": 3, "n": 4096},
        # the reproducible dot product of two long vectors, the library's headline call
        {"name": "ddot_2e28", "kind": "red", "type": "d", "op": "dot", "fold": 3, "n": 1 << 28},
        # the norm of a gradient or weight vector in FP32, an odd length
        {"name": "snrm2_100m", "kind": "red", "type": "s", "op": "nrm2", "fold": 3, "n": 100000007},
        # matrix-vector products of a dense solver: a square system of the benchmark's size ...
        {"name": "dgemv_n_4096", "kind": "gemv", "type": "d", "trans": "n", "fold": 3,
         "m": 4096, "n": 4096, "pad": 0},
        # ... and the transposed product of a matrix of odd sizes, as least squares applies it
        {"name": "dgemv_t_odd", "kind": "gemv", "type": "d", "trans": "t", "fold": 3,
         "m": 9001, "n": 3001, "pad": 0},
        # beamforming / adjoint operators: conjugate transpose of a complex FP32 matrix
        {"name": "cgemv_c_4096", "kind": "gemv", "type": "c", "trans": "c", "fold": 3,
         "m": 4096, "n": 4096, "pad": 0},
        # the plain binned matrix product at the benchmark's size
        {"name": "dgemm_2048", "kind": "gemm", "type": "d", "ta": "n", "tb": "n", "fold": 3,
         "m": 2048, "n": 2048, "k": 2048},
        # normal equations / covariance of a tall data matrix: X^T Y, few outputs, long sums
        {"name": "dgemm_gram", "kind": "gemm", "type": "d", "ta": "t", "tb": "n", "fold": 3,
         "m": 160, "n": 128, "k": 100000},
        # a layer's product in FP32 at sizes that fill no tile evenly
        {"name": "sgemm_odd", "kind": "gemm", "type": "s", "ta": "n", "tb": "t", "fold": 3,
         "m": 1000, "n": 1531, "k": 777},
        # complex FP64 block product with a conjugated operand (eigen- and scattering codes)
        {"name": "zgemm_c_768", "kind": "gemm", "type": "z", "ta": "c", "tb": "n", "fold": 3,
         "m": 768, "n": 768, "k": 768},
        # the int8-sliced product on the tensor cores at the benchmark's smaller size
        {"name": "int8_4096", "kind": "int8", "slices": 8, "m": 4096, "n": 4096, "k": 4096},
        # thousands of ragged dot products and hundreds of small products in one launch
        {"name": "batch_10k", "kind": "batch", "segments": 10000, "total": 1 << 26,
         "max_len": 1 << 20, "gemms": 512},
    ]


def _size(rng, lo, hi):
    """log-uniform in [lo, hi]; half of them odd or ragged, half multiples of 16"""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        v = (v + 8) // 16 * 16
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["red", "gemv", "gemv", "gemm", "gemm", "gemm", "int8", "batch"])
    fold = rng.choice([2, 3, 3, 3, 4])
    t = rng.choice("dszc")
    if kind == "red":
        return {"kind": kind, "type": t, "op": rng.choice(["sum", "dot", "nrm2"]), "fold": fold,
                "n": _size(rng, 1 << 10, (1 << 27) if t in "ds" else (1 << 26))}
    if kind == "gemv":
        trans = rng.choice("nt") if t in "ds" else rng.choice("ntc")
        while True:
            m, n = _size(rng, 64, 20000), _size(rng, 64, 20000)
            if (1 << 16) <= m * n <= (1 << 26):
                break
        return {"kind": kind, "type": t, "trans": trans, "fold": fold, "m": m, "n": n,
                "pad": rng.choice([0, 0, 1, 8])}
    if kind == "gemm":
        ta = rng.choice("nt") if t in "ds" else rng.choice("ntc")
        tb = rng.choice("nt") if t in "ds" else rng.choice("ntc")
        most = (1 << 31) if t in "ds" else (1 << 29)
        while True:
            m, n, k = _size(rng, 32, 4000), _size(rng, 32, 4000), _size(rng, 32, 100000)
            if (1 << 18) <= m * n * k <= most and k * max(m, n) <= 1 << 25:
                break
        return {"kind": kind, "type": t, "ta": ta, "tb": tb, "fold": fold, "m": m, "n": n, "k": k}
    if kind == "int8":
        return {"kind": kind, "slices": rng.choice([6, 7, 8, 10]), "m": _size(rng, 256, 4096),
                "n": _size(rng, 256, 4096), "k": _size(rng, 256, 4096)}
    return {"kind": kind, "segments": _size(rng, 100, 10000), "total": _size(rng, 1 << 20, 1 << 26),
            "max_len": 1 << 20, "gemms": rng.choice([0, 64, 512])}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, shape, t):
    """uniform(-1,1); complex elements as a trailing pair"""
    shape = tuple(shape) + ((2,) if t in "zc" else ())
    return torch.rand(shape, generator=g, dtype=_REAL[t], device="cuda").mul_(2).sub_(1)


def _scalar(t, re, im):
    return (ctypes.c_double * 2)(re, im) if t == "z" else (ctypes.c_float * 2)(re, im) \
        if t == "c" else re


_ALPHA, _ALPHA_I = 1.5, -0.25


def _scalars(t):
    a, b = _scalar(t, _ALPHA, _ALPHA_I), _scalar(t, 0.0, 0.0)
    return a, b, (ctypes.addressof(a) if t in "zc" else a), (ctypes.addressof(b) if t in "zc" else b)


class _Plan:
    """a batch plan and the memory it refers to"""

    def __init__(self, case, seed):
        g = _gen(seed)
        # the shapes belong to the case (the same ragged problem with other data)
        r = torch.Generator().manual_seed(case["segments"] * 1000003 + case["total"])
        S, total = case["segments"], case["total"]
        lens = torch.exp(torch.rand(S, generator=r, dtype=torch.float64) * math.log(case["max_len"]))
        lens = torch.clamp((lens * (total / float(lens.sum()))).to(torch.int64), 1, case["max_len"])
        offs = torch.cumsum(lens, 0) - lens
        n = int(lens.sum())
        self.lens, self.offs = lens.to(torch.int32), offs
        self.x = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
        self.y = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
        self.results = torch.zeros(S, dtype=torch.float64, device="cuda")
        G = case["gemms"]
        self.mnk = [tuple(int(v) for v in torch.randint(16, 257, (3,), generator=r))
                    for _ in range(G)]
        self.A = _uniform(g, (sum(m * k for m, n_, k in self.mnk) + 1,), "d")
        self.B = _uniform(g, (sum(k * n_ for m, n_, k in self.mnk) + 1,), "d")
        self.C = torch.zeros(sum(m * n_ for m, n_, k in self.mnk) + 1, dtype=torch.float64,
                             device="cuda")
        inst = (rb.DgemmInstance * max(G, 1))()
        a = b = c = 0
        for i, (m, n_, k) in enumerate(self.mnk):
            d = inst[i]
            d.order, d.transa, d.transb = b"r", b"n", b"n"
            d.m, d.n, d.k, d.alpha, d.beta = m, n_, k, 1.0, 0.0
            d.A, d.lda = self.A.data_ptr() + 8 * a, k
            d.B, d.ldb = self.B.data_ptr() + 8 * b, n_
            d.C, d.ldc = self.C.data_ptr() + 8 * c, n_
            a, b, c = a + m * k, b + k * n_, c + m * n_
        self.plan = rb.lib.rb_batch_plan_create(
            3, S, self.offs.data_ptr(), self.lens.data_ptr(), self.x.data_ptr(),
            self.y.data_ptr(), self.results.data_ptr(), None, G, ctypes.addressof(inst))
        rb.check()

    def __del__(self):
        if getattr(self, "plan", None):
            rb.lib.rb_batch_plan_destroy(self.plan)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "plan": _Plan(case, seed)}
    g = _gen(seed)
    if kind == "red":
        t, n = case["type"], case["n"]
        shape = (n, 2) if t in "zc" else (n,)
        s = {"kind": kind, "op": case["op"], "type": t, "fold": case["fold"], "n": n,
             "x": torch.randn(shape, generator=g, dtype=_REAL[t], device="cuda")}
        if case["op"] == "dot":
            s["y"] = torch.randn(shape, generator=g, dtype=_REAL[t], device="cuda")
        if t in "zc" and case["op"] != "nrm2":
            s["out"] = torch.zeros(2, dtype=_REAL[t], device="cuda")
        return s
    if kind == "gemv":
        t, m, n = case["type"], case["m"], case["n"]
        lda = n + case["pad"]
        s = {"kind": kind, "type": t, "trans": case["trans"], "fold": case["fold"], "m": m, "n": n,
             "lda": lda, "scalars": _scalars(t), "A": _uniform(g, (m, lda), t)}
        nt = case["trans"] == "n"
        s["x"] = _uniform(g, (n if nt else m,), t)
        s["y"] = torch.zeros((m if nt else n,) + ((2,) if t in "zc" else ()), dtype=_REAL[t],
                             device="cuda")
        return s
    if kind == "gemm":
        t, m, n, k = case["type"], case["m"], case["n"], case["k"]
        s = {"kind": kind, "type": t, "ta": case["ta"], "tb": case["tb"], "fold": case["fold"],
             "m": m, "n": n, "k": k, "scalars": _scalars(t)}
        s["A"] = _uniform(g, (m, k) if case["ta"] == "n" else (k, m), t)
        s["B"] = _uniform(g, (k, n) if case["tb"] == "n" else (n, k), t)
        s["C"] = torch.zeros((m, n) + ((2,) if t in "zc" else ()), dtype=_REAL[t], device="cuda")
        return s
    m, n, k = case["m"], case["n"], case["k"]

    def wide(rows, cols):
        # mantissas in [1, 2), exponents in [-20, 20], random signs
        v = 1 + torch.rand(rows, cols, generator=g, dtype=torch.float64, device="cuda")
        e = torch.randint(-20, 21, (rows, cols), generator=g, device="cuda")
        sg = torch.randint(0, 2, (rows, cols), generator=g, device="cuda") * 2 - 1
        return torch.ldexp(v * sg, e)

    return {"kind": kind, "slices": case["slices"], "m": m, "n": n, "k": k, "A": wide(m, k),
            "B": wide(k, n), "C": torch.zeros(m, n, dtype=torch.float64, device="cuda")}


def run(s):
    kind = s["kind"]
    if kind == "red":
        t, op, x = s["type"], s["op"], s["x"]
        if op == "nrm2":
            name = {"d": "dnrm2", "s": "snrm2", "z": "dznrm2", "c": "scnrm2"}[t]
            return rb.call("reproBLAS_r" + name, s["fold"], s["n"], x, 1)
        if t in "ds":
            if op == "sum":
                return rb.call("reproBLAS_r%ssum" % t, s["fold"], s["n"], x, 1)
            return rb.call("reproBLAS_r%sdot" % t, s["fold"], s["n"], x, 1, s["y"], 1)
        if op == "sum":
            rb.call("reproBLAS_r%ssum_sub" % t, s["fold"], s["n"], x, 1, s["out"])
        else:
            rb.call("reproBLAS_r%sdotc_sub" % t, s["fold"], s["n"], x, 1, s["y"], 1, s["out"])
        return s["out"]
    if kind == "gemv":
        _, _, alpha, beta = s["scalars"]
        rb.call("reproBLAS_r%sgemv" % s["type"], s["fold"], "r", s["trans"], s["m"], s["n"], alpha,
                s["A"], s["lda"], s["x"], 1, beta, s["y"], 1)
        return s["y"]
    if kind == "gemm":
        _, _, alpha, beta = s["scalars"]
        m, n, k = s["m"], s["n"], s["k"]
        rb.call("reproBLAS_r%sgemm" % s["type"], s["fold"], "r", s["ta"], s["tb"], m, n, k, alpha,
                s["A"], k if s["ta"] == "n" else m, s["B"], n if s["tb"] == "n" else k, beta,
                s["C"], n)
        return s["C"]
    if kind == "int8":
        m, n, k = s["m"], s["n"], s["k"]
        rb.call("rb_dgemm_int8", 3, "r", "n", "n", m, n, k, 1.0, s["A"], k, s["B"], n, 0.0,
                s["C"], n, s["slices"])
        return s["C"]
    p = s["plan"]
    rb.lib.rb_batch_plan_run(p.plan, None)
    rb.check()
    return {"dots": p.results, "products": p.C}


def exact(case, seed):
    s = prepare(case, seed)
    kind = s["kind"]

    def wide(v):
        v = v.double()
        return torch.view_as_complex(v) if case["type"] in "zc" else v

    def narrow(v):
        return torch.view_as_real(v) if v.is_complex() else v

    if kind == "red":
        x = wide(s["x"])
        if s["op"] == "nrm2":
            return float(torch.linalg.vector_norm(x))
        v = x.sum() if s["op"] == "sum" else torch.vdot(x, wide(s["y"]))
        return narrow(v) if v.is_complex() else float(v)
    if kind in ("gemv", "gemm"):
        def op(a, tr):
            return a if tr == "n" else a.T if tr == "t" else a.conj().T
        alpha = complex(_ALPHA, _ALPHA_I) if case["type"] in "zc" else _ALPHA
        A = wide(s["A"])
        if kind == "gemv":
            return narrow(op(A[:, :s["n"]], s["trans"]) @ (alpha * wide(s["x"])))
        return narrow(alpha * (op(A, s["ta"]) @ op(wide(s["B"]), s["tb"])))
    if kind == "int8":
        return s["A"] @ s["B"]
    p = s["plan"]
    dots = torch.segment_reduce(p.x * p.y, "sum", lengths=p.lens.long().cuda())
    C = torch.zeros_like(p.C)
    a = b = c = 0
    for m, n, k in p.mnk:
        C[c:c + m * n] = (p.A[a:a + m * k].view(m, k) @ p.B[b:b + k * n].view(k, n)).reshape(-1)
        a, b, c = a + m * k, b + k * n, c + m * n
    return {"dots": dots, "products": C}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # expected sizes of the 512 (or fewer) products: m, n, k uniform in 16..256
        e = 136
        return {"bytes": 16 * case["total"] + 8 * case["segments"] + 24 * e * e * case["gemms"],
                "flops": 2 * case["total"] + 2 * e ** 3 * case["gemms"]}
    if kind == "int8":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    t = case["type"]
    size = {"d": 8, "s": 4, "z": 16, "c": 8}[t]
    mul = 4 if t in "zc" else 1
    if kind == "red":
        n = case["n"]
        return {"bytes": size * n * (2 if case["op"] == "dot" else 1),
                "flops": (1 if case["op"] == "sum" else 2) * n * mul}
    m, n = case["m"], case["n"]
    if kind == "gemv":
        return {"bytes": size * (m * n + m + n), "flops": 2 * m * n * mul}
    k = case["k"]
    return {"bytes": size * (m * k + k * n + m * n), "flops": 2 * m * n * k * mul}
