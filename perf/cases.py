"""Workloads of the library that its speed is judged by.

Each case is one call that a user's program makes through the public entry
points (``gemm_avx512f_b200.blas`` and the grouped calls of the C ABI) on
matrices of its own, with the sizes, value distributions and options of the
library's own configurations (``gemm_avx512f_b200/inputs.py``), plus tiny,
ragged and padded ones.  ``draw`` gives further cases of the same ranges.

All matrices are column-major.  ``pad`` is added to every leading dimension
(a sub-matrix of a larger array; an odd pad also breaks 16-byte alignment of
the columns).  Calls are issued on one stream of the program's own, as the
library asks of a thread.  With beta != 0 the output is updated in place on
every pass; |beta| < 1 keeps it bounded.
"""
import ctypes as C
import math

import numpy as np
import torch

from gemm_avx512f_b200 import _lib, blas

_STREAM = None


def _stream():
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


# ------------------------------------------------------------------- cases --
def _gemm(op, ta, tb, m, n, k, method="default", alpha=1.0, beta=0.0, pad=0, phi=0.0, name=None):
    c = {"op": op, "ta": ta, "tb": tb, "m": m, "n": n, "k": k, "method": method,
         "alpha": alpha, "beta": beta, "pad": pad, "phi": phi}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest call: a product of a few dozen rows inside a larger
        # program (padded leading dimensions); latency is all there is.
        _gemm("dgemm", "T", "N", 48, 40, 64, "fp64", 1.5, 0.5, 3, name="dgemm small"),
        # The plain DGEMM configuration (alpha 1.5, beta 0.5).
        _gemm("dgemm", "N", "N", 1024, 1024, 1024, "fp64", 1.5, 0.5, name="dgemm 1024"),
        # An ordinary product of a program whose sizes are its data's: odd
        # sizes, an odd leading dimension, B transposed.
        _gemm("dgemm", "N", "T", 2501, 1777, 1999, "fp64", 1.0, 0.0, 2, name="dgemm ragged"),
        # The largest: FP64 accuracy from the INT8 tensor cores, 8192^3 with
        # log-normally spread magnitudes.
        _gemm("dgemm", "N", "N", 8192, 8192, 8192, "ozaki", 1.0, 0.0, 0, 1.0, name="dgemm ozaki 8192"),
        # sgemm_'s default method (FP32 on the CUDA cores) at its middle size.
        _gemm("sgemm", "N", "N", 4096, 4096, 4096, "fp32", 1.0, 0.0, name="sgemm fp32 4096"),
        # Split SGEMM at its smallest configured square, transposed A.
        _gemm("sgemm", "T", "N", 2048, 2048, 2048, "tf32x3", 1.0, 0.0, name="sgemm tf32x3 2048"),
        # The rectangular SGEMM configuration (few columns, long K).
        _gemm("sgemm", "N", "T", 8192, 256, 8192, "bf16x3", 1.0, 0.0, name="sgemm bf16x3 rect"),
        # Complex 3M products: the configured complex128 square, and a ragged
        # complex64 one with conjugated A.
        _gemm("zgemm3m", "N", "N", 2048, 2048, 2048, name="zgemm3m 2048"),
        _gemm("cgemm3m", "C", "N", 1900, 1300, 2100, alpha=0.5, beta=0.5, name="cgemm3m ragged"),
        # Triangular solve against a block of right-hand sides (a quarter of
        # the configured order and right-hand sides).
        {"name": "dtrsm 4096", "op": "dtrsm", "side": "L", "uplo": "L", "ta": "N", "diag": "N",
         "m": 4096, "n": 1024, "alpha": 1.0, "pad": 0, "method": "fp64"},
        # Many unrelated products kept as a plan: the grouped configuration's
        # distribution, a quarter of its problems.
        {"name": "grouped 1024", "op": "grouped", "count": 1024, "plan": True, "lo": 16,
         "hi": 1024, "mix": "df", "beta": 0.0},
        # The drop-in symbol on a caller's own (pageable) host arrays.
        _gemm("dgemm_host", "N", "N", 1200, 900, 1500, "fp64", 1.0, 0.5, name="dgemm_ host"),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]; every second one as
    it falls, the others rounded to 16 or 64 (sizes people choose)."""
    v = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    r = rng.random()
    if r < 0.25:
        v = v // 16 * 16
    elif r < 0.5 and v >= 64:
        v = v // 64 * 64
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["dgemm", "dgemm", "ozaki", "fp32", "tf32", "tf32x3", "bf16x3", "zgemm3m",
                       "cgemm3m", "dtrsm", "grouped", "host"])
    nt = lambda: rng.choice("NT")  # noqa: E731
    beta = rng.choice([0.0, 0.0, 0.5])
    alpha = rng.choice([1.0, 1.0, 1.5, -0.5])
    pad = rng.choice([0, 0, 0, 1, 4])
    if kind == "dgemm":
        return _gemm("dgemm", nt(), nt(), *(_log_int(rng, 24, 4096) for _ in range(3)), "fp64",
                     alpha, beta, pad)
    if kind == "ozaki":
        return _gemm("dgemm", nt(), nt(), *(_log_int(rng, 700, 8192) for _ in range(3)), "ozaki",
                     alpha, beta, pad, rng.choice([0.1, 1.0, 4.0]))
    if kind == "fp32":
        return _gemm("sgemm", nt(), nt(), *(_log_int(rng, 128, 8192) for _ in range(3)), "fp32",
                     alpha, beta, pad)
    if kind in ("tf32", "tf32x3", "bf16x3"):
        return _gemm("sgemm", nt(), nt(), *(_log_int(rng, 200, 8192) for _ in range(3)), kind,
                     alpha, beta, pad)
    if kind == "zgemm3m":
        return _gemm("zgemm3m", rng.choice("NTCR"), rng.choice("NTCR"),
                     *(_log_int(rng, 48, 2048) for _ in range(3)), "default", alpha, beta, pad)
    if kind == "cgemm3m":
        return _gemm("cgemm3m", rng.choice("NTCR"), rng.choice("NTCR"),
                     *(_log_int(rng, 48, 3072) for _ in range(3)), "default", alpha, beta, pad)
    if kind == "dtrsm":
        return {"op": "dtrsm", "side": rng.choice("LR"), "uplo": rng.choice("LU"),
                "ta": nt(), "diag": rng.choice("NNU"), "m": _log_int(rng, 64, 4096),
                "n": _log_int(rng, 64, 4096), "alpha": alpha, "pad": pad,
                "method": rng.choice(["fp64", "fp64", "ozaki"])}
    if kind == "grouped":
        lo = rng.choice([16, 24, 40])
        return {"op": "grouped", "count": _log_int(rng, 32, 1024), "plan": rng.random() < 0.6,
                "lo": lo, "hi": rng.choice([256, 640, 1024]),
                "mix": rng.choice(["df", "df", "d", "f", "dfz"]), "beta": beta}
    return _gemm("dgemm_host", nt(), nt(), *(_log_int(rng, 64, 2048) for _ in range(3)), "fp64",
                 alpha, beta, pad)


# ------------------------------------------------------------------ inputs --
_REAL = {"dgemm": torch.float64, "dgemm_host": torch.float64, "sgemm": torch.float32}
_CPLX = {"zgemm3m": torch.complex128, "cgemm3m": torch.complex64}


def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _uniform(n, dtype, g):
    """n values U[-1, 1) (real and imaginary part each for complex types)."""
    if dtype.is_complex:
        rt = torch.float64 if dtype == torch.complex128 else torch.float32
        x = torch.rand(2 * n, dtype=rt, device="cuda", generator=g).mul_(2).sub_(1)
        return torch.view_as_complex(x.view(n, 2))
    return torch.rand(n, dtype=dtype, device="cuda", generator=g).mul_(2).sub_(1)


def _shapes(case):
    """(rows, cols) of A and B as stored, and their leading dimensions."""
    keep = "NR"
    ar, ac = (case["m"], case["k"]) if case["ta"] in keep else (case["k"], case["m"])
    br, bc = (case["k"], case["n"]) if case["tb"] in keep else (case["n"], case["k"])
    p = case["pad"]
    return (ar, ac, ar + p), (br, bc, br + p)


def _grouped_shapes(case):
    """(dtype, ta, tb, m, n, k) per problem: M, N, K log-uniform in [lo, hi],
    as the grouped configuration draws them; the mix names the types in turn."""
    rng = np.random.default_rng([3, case["count"], case["lo"], case["hi"]])
    cnt, lo, hi = case["count"], case["lo"], case["hi"]
    dims = np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), (cnt, 3)))).astype(int)
    dims = np.clip(dims, lo, hi)
    trans = rng.integers(0, 2, (cnt, 2))
    out = []
    for i in range(cnt):
        dt = "dfz".index(case["mix"][i % len(case["mix"])])
        m, n, k = (int(v) for v in dims[i])
        if dt == 2:  # complex problems are the smaller part of such a batch
            m, n, k = min(m, 256), min(n, 256), min(k, 256)
        out.append((dt, "NT"[trans[i, 0]], "NT"[trans[i, 1]], m, n, k))
    return out


_GT = (torch.float64, torch.float32, torch.complex128)


def _grouped_inputs(case, seed):
    """Flat A, B, C buffers per type and each problem's offsets in them."""
    shapes = _grouped_shapes(case)
    size = [[0, 0, 0] for _ in _GT]
    probs = []
    for dt, ta, tb, m, n, k in shapes:
        offs = tuple(size[dt])
        for j, v in enumerate((m * k, k * n, m * n)):
            size[dt][j] += (v + 31) // 32 * 32  # every matrix starts on a 128-byte boundary
        probs.append((dt, ta, tb, m, n, k, offs))
    bufs = [[_uniform(max(1, s), t, _gen(seed, 10 * d + j)) for j, s in enumerate(size[d])]
            for d, t in enumerate(_GT)]
    return probs, bufs


def _trsm_inputs(case, seed):
    """Triangle with off-diagonal U[-1,1) and a dominant diagonal n + U[0,1)
    (unit solves: off-diagonal scaled by 1/n instead), and right-hand sides."""
    m, n, p = case["m"], case["n"], case["pad"]
    na = m if case["side"] == "L" else n
    a = _uniform((na + p) * na, torch.float64, _gen(seed, 1)).view(na, na + p)  # [col][row]
    if case["diag"] == "U":
        a.mul_(1.0 / na)
    else:
        a.diagonal().abs_().add_(na)
    b = _uniform((m + p) * n, torch.float64, _gen(seed, 2)).view(n, m + p)
    return a, b


def prepare(case, seed):
    op = case["op"]
    if op == "grouped":
        probs, bufs = _grouped_inputs(case, seed)
        arr = (_lib.GemmProblem * len(probs))()
        for i, (dt, ta, tb, m, n, k, offs) in enumerate(probs):
            es = bufs[dt][0].element_size()
            pa, pb, pc = (bufs[dt][j].data_ptr() + offs[j] * es for j in range(3))
            arr[i] = _lib.GemmProblem(dt, ta.encode(), tb.encode(), m, n, k, 1.0, case["beta"],
                                      pa, m if ta == "N" else k, pb, k if tb == "N" else n, pc, m,
                                      0.0, 0.0)
        st = {"case": case, "bufs": bufs, "arr": arr, "stream": _stream(),
              "out": [bufs[d][2] for d in sorted({p[0] for p in probs})]}
        if case["plan"]:
            st["plan"] = _Plan(arr)
        return st
    if op == "dtrsm":
        a, b = _trsm_inputs(case, seed)
        return {"case": case, "a": a, "b": b, "x": torch.empty_like(b), "stream": _stream()}
    dt = _CPLX.get(op) or _REAL[op]
    (ar, ac, lda), (br, bc, ldb) = _shapes(case)
    ldc = case["m"] + case["pad"]
    a = _uniform(lda * ac, dt, _gen(seed, 1))
    b = _uniform(ldb * bc, dt, _gen(seed, 2))
    if case["phi"]:
        for i, x in enumerate((a, b)):
            g = torch.randn(x.numel(), dtype=dt, device="cuda", generator=_gen(seed, 3 + i))
            x.mul_(g.mul_(case["phi"]).exp_())
    # an output that is only written (beta = 0) starts at zero, as a caller's does
    c = (_uniform(ldc * case["n"], dt, _gen(seed, 5)) if case["beta"]
         else torch.zeros(ldc * case["n"], dtype=dt, device="cuda"))
    st = {"case": case, "a": a, "b": b, "c": c, "lda": lda, "ldb": ldb, "ldc": ldc,
          "stream": _stream()}
    if op == "dgemm_host":
        st.update({x: st[x].cpu().numpy() for x in "abc"})
    return st


class _Plan:
    """A grouped plan that is destroyed with the state that holds it."""

    def __init__(self, arr):
        self.handle, self.destroy = C.c_void_p(), _lib.lib().b2_grouped_plan_destroy
        _lib.check(_lib.lib().b2_grouped_plan_create(len(arr), arr, C.byref(self.handle)),
                   "b2_grouped_plan_create")

    def __del__(self):
        self.destroy(self.handle)


# --------------------------------------------------------------- one pass --
def run(st):
    case, s = st["case"], st["stream"]
    op = case["op"]
    if op == "grouped":
        L = _lib.lib()
        if "plan" in st:
            _lib.check(L.b2_grouped_plan_launch(st["plan"].handle, s.cuda_stream),
                       "b2_grouped_plan_launch")
        else:
            _lib.check(L.b2_gemm_grouped(len(st["arr"]), st["arr"], s.cuda_stream),
                       "b2_gemm_grouped")
        return st["out"]
    if op == "dtrsm":
        # solved in place in a copy: the right-hand sides are still needed
        with torch.cuda.stream(s):
            st["x"].copy_(st["b"])
        ld = case["m"] + case["pad"]
        na = case["m"] if case["side"] == "L" else case["n"]
        blas.dtrsm_device(case["side"], case["uplo"], case["ta"], case["diag"], case["m"],
                          case["n"], case["alpha"], st["a"], na + case["pad"], st["x"], ld,
                          update=case["method"], stream=s)
        return st["x"]
    args = (case["ta"], case["tb"], case["m"], case["n"], case["k"], case["alpha"], st["a"],
            st["lda"], st["b"], st["ldb"], case["beta"], st["c"], st["ldc"])
    if op == "dgemm":
        return blas.dgemm_device(*args, method=case["method"], stream=s)
    if op == "sgemm":
        return blas.sgemm_device(*args, method=case["method"], stream=s)
    if op == "zgemm3m":
        return blas.zgemm3m_device(*args, stream=s)
    if op == "cgemm3m":
        return blas.cgemm3m_device(*args, stream=s)
    return blas.dgemm(*args)


# -------------------------------------------------------------------- work --
def work(case):
    op = case["op"]
    if op == "grouped":
        by = fl = 0
        for dt, _, _, m, n, k in _grouped_shapes(case):
            by += (8, 4, 16)[dt] * (m * k + k * n + 2 * m * n)
            fl += (2, 2, 6)[dt] * m * n * k
        return {"bytes": by, "flops": fl}
    if op == "dtrsm":
        m, n = case["m"], case["n"]
        na, nv = (m, n) if case["side"] == "L" else (n, m)
        return {"bytes": 8 * (na * (na + 1) // 2 + 2 * na * nv), "flops": na * na * nv}
    # C counts as read even for beta = 0: a NaN already in C stays there.
    m, n, k = case["m"], case["n"], case["k"]
    es = {"sgemm": 4, "cgemm3m": 8, "zgemm3m": 16}.get(op, 8)
    return {"bytes": es * (m * k + k * n + 2 * m * n),
            "flops": (6 if op in _CPLX else 2) * m * n * k}


# ------------------------------------------------------------------- exact --
def _op(x, t):
    return {"N": x, "T": x.t(), "C": x.t().conj(), "R": x.conj()}[t]


def exact(case, seed):
    op = case["op"]
    if op == "grouped":
        probs, bufs = _grouped_inputs(case, seed)
        up = lambda x: x.to(torch.complex128 if x.dtype.is_complex else torch.float64)  # noqa: E731
        out = {}
        for dt, ta, tb, m, n, k, offs in probs:
            A, B, Cm = bufs[dt]
            a = A[offs[0]:offs[0] + m * k].view(*((k, m) if ta == "N" else (m, k)))
            b = B[offs[1]:offs[1] + k * n].view(*((n, k) if tb == "N" else (k, n)))
            if dt not in out:
                out[dt] = up(Cm)
            c = out[dt][offs[2]:offs[2] + m * n].view(n, m)
            c.mul_(case["beta"]).add_(_op(up(b).t(), tb).t() @ _op(up(a).t(), ta).t())
        return [out[d] for d in sorted(out)]
    if op == "dtrsm":
        a, b = _trsm_inputs(case, seed)
        m, n = case["m"], case["n"]
        na = m if case["side"] == "L" else n
        A = a[:, :na].t()
        A = torch.triu(A) if case["uplo"] == "U" else torch.tril(A)
        upper = case["uplo"] == "U"
        if case["ta"] == "T":
            A, upper = A.t(), not upper
        B = b[:, :m].t() * case["alpha"]
        X = torch.linalg.solve_triangular(A, B, upper=upper, left=case["side"] == "L",
                                          unitriangular=case["diag"] == "U")
        out = b.clone()
        out[:, :m] = X.t()
        return out
    st = prepare(case, seed)
    if op == "dgemm_host":
        st.update({x: torch.from_numpy(st[x]).cuda() for x in "abc"})
    wide = torch.complex128 if op in _CPLX else torch.float64
    (ar, ac, lda), (br, bc, ldb) = _shapes(case)
    a = _op(st["a"].view(ac, lda)[:, :ar].t().to(wide), case["ta"])
    b = _op(st["b"].view(bc, ldb)[:, :br].t().to(wide), case["tb"])
    out = st["c"].to(wide).clone()
    c = out.view(case["n"], st["ldc"])[:, :case["m"]]
    c.mul_(case["beta"]).add_((a @ b).t(), alpha=case["alpha"])
    return out.cpu().numpy() if op == "dgemm_host" else out
