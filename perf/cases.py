"""The library's performance cases: what its callers have it do, through its public entry points.

A case is a dict of plain values; its "op" says which entry point it takes:

  gemm   api.gemm(transa, transb, ...)                     C = alpha op(A) op(B) + beta C
  syrk   api.syrk(uplo, trans, ...)                        one triangle of C
  lu     api.getrf, then api.getrs for nrhs > 0            FP64, BOLA's rounding
  chol   api.potrf, then api.potrs for nrhs > 0            FP64, BOLA's rounding
  trsm   api.trsm(side, uplo, trans, diag, ...)            FP64, BOLA's rounding
  mixed  bola_dgesv_mixed_ctx / bola_dposv_mixed_ctx       low-precision factor, FP64 refinement
  batch  batch.Batch.solve                                 many small systems in one launch

Matrices are column-major.  Routines that overwrite an operand get a fresh
copy of it in each pass, as a program that assembles a new matrix into the
same buffer does.  Mixed solves have condition numbers up to 1e4: two answers
of backward error 1e-14 then agree to about 1e-10.  (For a worse-conditioned
system two equally good answers differ by more; the kernels that run are
those of factor kinds 2 and 3, which are both here.)  The solve server is not
a case of its own: its requests go through the mixed and batched solves below.
"""
import ctypes
import math

import numpy as np
import torch

from bola_gb300 import _lib, api
from bola_gb300.batch import Batch

F64 = torch.float64


def listed():
    return [
        # A block update of a small assembly or of a caller's own blocked algorithm: launch latency counts.
        {"name": "gemm-small-nt", "op": "gemm", "ta": "N", "tb": "T", "m": 61, "n": 48, "k": 75, "alpha": -1.0, "beta": 1.0},
        # The size that BOLA's own benchmark starts with.
        {"name": "gemm-nn-1024", "op": "gemm", "ta": "N", "tb": "N", "m": 1024, "n": 1024, "k": 1024, "alpha": 1.0, "beta": 1.0},
        # Normal equations and projections: transposed A, sizes that divide by nothing.
        {"name": "gemm-tn-ragged", "op": "gemm", "ta": "T", "tb": "N", "m": 2051, "n": 1530, "k": 777, "alpha": 1.0, "beta": 0.0},
        # A model with some hundred unknowns, solved again and again.
        {"name": "lu-solve-200", "op": "lu", "m": 200, "n": 200, "nrhs": 3},
        # The size that BOLA's LU benchmark starts with.
        {"name": "lu-1024", "op": "lu", "m": 1024, "n": 1024, "nrhs": 0},
        # The large plain factorisation (BOLA's largest benchmark).
        {"name": "lu-4096", "op": "lu", "m": 4096, "n": 4096, "nrhs": 0},
        # A covariance or kernel matrix kept as its upper triangle, solved for a few vectors.
        {"name": "chol-u-777", "op": "chol", "uplo": "U", "n": 777, "nrhs": 9},
        # The large plain Cholesky.
        {"name": "chol-l-4096", "op": "chol", "uplo": "L", "n": 4096, "nrhs": 0},
        # Unit-lower solve of many right-hand sides with a large factor.
        {"name": "trsm-llnu-4096", "op": "trsm", "side": "L", "uplo": "L", "ta": "N", "diag": "U", "m": 4096, "n": 1024, "alpha": 1.0},
        # The headline solve: n=8192, 16 right-hand sides, to a backward error of 1e-14.
        {"name": "mixed-lu-8192", "op": "mixed", "spd": False, "n": 8192, "nrhs": 16, "kind": 2, "logk": 2.0},
        # A request of the size that a solve server sees most, SPD.
        {"name": "mixed-spd-1500", "op": "mixed", "spd": True, "n": 1500, "nrhs": 5, "kind": 2, "logk": 3.0},
        # Many uneven small systems, half LU and half Cholesky, replayed as a graph.
        {"name": "batch-4000", "op": "batch", "count": 4000, "nmin": 8, "nmax": 256, "rmax": 8, "graph": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["gemm", "gemm", "syrk", "lu", "lu", "chol", "trsm", "trsm", "mixed", "mixed", "batch"])
    if op == "gemm":
        c = {"op": op, "ta": rng.choice("NT"), "tb": rng.choice("NT"), "m": _log(rng, 16, 3000), "n": _log(rng, 16, 3000),
             "k": _log(rng, 16, 3000), "alpha": rng.choice([1.0, -1.0, 0.75]), "beta": rng.choice([0.0, 1.0, 0.5])}
    elif op == "syrk":
        uplo, trans = rng.choice(["LN", "UT"])
        c = {"op": op, "uplo": uplo, "trans": trans, "n": _log(rng, 16, 2000), "k": _log(rng, 16, 2000), "alpha": -1.0, "beta": 1.0}
    elif op == "lu":
        n = _log(rng, 24, 4000)
        nrhs = rng.choice([0, 0, 1, 5, 32])
        m = n if nrhs else min(4096, n + rng.choice([0, 0, rng.randint(1, 600)]))
        c = {"op": op, "m": m, "n": n, "nrhs": nrhs}
    elif op == "chol":
        c = {"op": op, "uplo": rng.choice("UL"), "n": _log(rng, 24, 4000), "nrhs": rng.choice([0, 0, 1, 5, 32])}
    elif op == "trsm":
        side = rng.choice("LR")
        big, small = _log(rng, 24, 3000), _log(rng, 8, 1000)
        c = {"op": op, "side": side, "uplo": rng.choice("LU"), "ta": rng.choice("NT"), "diag": rng.choice("NU"),
             "m": big if side == "L" else small, "n": small if side == "L" else big, "alpha": rng.choice([1.0, -0.5])}
    elif op == "mixed":
        c = {"op": op, "spd": rng.random() < 0.3, "n": _log(rng, 260, 8000), "nrhs": rng.randint(1, 32),
             "kind": rng.choice([2, 2, 3]), "logk": round(rng.uniform(1.0, 4.0), 3)}
    else:
        nmin = _log(rng, 4, 64)
        c = {"op": op, "count": _log(rng, 50, 3900), "nmin": nmin, "nmax": rng.randint(nmin, 256), "rmax": rng.randint(1, 8),
             "graph": rng.random() < 0.5}
    return c


# ---- inputs ------------------------------------------------------------------

class _Draw:
    """Seeded numbers on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) & 0x7FFFFFFF)

    def uniform(self, rows, cols, lo=-1.0, hi=1.0):
        """rows x cols, uniform in [lo, hi), a column-major matrix."""
        u = torch.rand(cols, rows, dtype=F64, device="cuda", generator=self.g)
        return u.mul_(hi - lo).add_(lo).t()

    def _rotate(self, M):
        """M with a random orthogonal matrix applied to its rows: random signs, then a circulant whose spectrum has
        unit modulus, twice."""
        n = M.shape[0]
        for _ in range(2):
            sign = torch.randint(0, 2, (n, 1), device="cuda", generator=self.g).to(F64) * 2 - 1
            phase = torch.rand(n // 2 + 1, 1, dtype=F64, device="cuda", generator=self.g) * (2 * math.pi)
            phase[0] = 0
            if n % 2 == 0:
                phase[-1] = 0
            M = torch.fft.irfft(torch.fft.rfft(M * sign, dim=0) * torch.polar(torch.ones_like(phase), phase), n=n, dim=0)
        return M

    def general(self, n, logk):
        """Q1 diag(sigma) Q2, sigma geometric from 1 to 10^-logk."""
        sigma = torch.logspace(0.0, -logk, n, dtype=F64, device="cuda")
        return self._rotate(self._rotate(torch.diag(sigma)).t())

    def spd(self, n, logk):
        """Q diag(sigma) Q^T, exactly symmetric."""
        sigma = torch.logspace(0.0, -0.5 * logk, n, dtype=F64, device="cuda")
        H = self._rotate(torch.diag(sigma))
        S = H @ H.t()
        return (S + S.t()) * 0.5


def _flat(M):
    """Column-major storage of M as a flat tensor of its own."""
    return M.t().contiguous().reshape(-1)


def _dense(v, m, n):
    """The m x n matrix whose column-major storage v is."""
    return v.reshape(n, m).t()


def _triangle(d, m, uplo, diag):
    """A triangular factor of moderate growth; the other triangle holds what a solve must not read."""
    A = d.uniform(m, m) * (1.0 / math.sqrt(m))
    if diag == "N":
        A = A + torch.diag(1.0 + d.uniform(m, 1, 0.0, 1.0).reshape(-1))
    return A


def _inputs(case, seed):
    d, op = _Draw(seed), case["op"]
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        a = d.uniform(m, k, 0.0, 1.0) if case["ta"] == "N" else d.uniform(k, m, 0.0, 1.0)
        b = d.uniform(k, n, 0.0, 1.0) if case["tb"] == "N" else d.uniform(n, k, 0.0, 1.0)
        return {"a": a, "b": b, "c": d.uniform(m, n, 0.0, 1.0)}
    if op == "syrk":
        n, k = case["n"], case["k"]
        a = d.uniform(n, k) if case["trans"] == "N" else d.uniform(k, n)
        c = d.uniform(n, n)
        return {"a": a, "c": c + c.t()}
    if op == "lu":
        return {"a": d.uniform(case["m"], case["n"]), "b": d.uniform(case["n"], max(1, case["nrhs"]))}
    if op == "chol":
        n = case["n"]
        h = d.uniform(n, n)
        return {"a": h @ h.t() / n + torch.eye(n, dtype=F64, device="cuda"), "b": d.uniform(n, max(1, case["nrhs"]))}
    if op == "trsm":
        return {"a": _triangle(d, case["m"] if case["side"] == "L" else case["n"], case["uplo"], case["diag"]),
                "b": d.uniform(case["m"], case["n"])}
    if op == "mixed":
        n = case["n"]
        a = d.spd(n, case["logk"]) if case["spd"] else d.general(n, case["logk"])
        x = d.uniform(n, case["nrhs"])
        return {"a": a, "b": a @ x}
    assert op == "batch", op
    ns, nrhs, kinds = _sizes(case)
    return {"ns": ns, "nrhs": nrhs, "kinds": kinds, "draw": d}


def _sizes(case):
    """A batch's sizes: uniform, the same for every seed of the values."""
    rng = np.random.default_rng(case["count"])
    ns = rng.integers(case["nmin"], case["nmax"] + 1, size=case["count"]).astype(np.int32)
    nrhs = rng.integers(1, case["rmax"] + 1, size=case["count"]).astype(np.int32)
    return ns, nrhs, (np.arange(case["count"]) % 2).astype(np.int32)


def _fill(ns, nrhs, kinds, d, a_view, b_view):
    """Even systems: uniform[-1,1) + n I; odd ones: H H^T / n + I with H uniform."""
    a, b = d.uniform(int((ns.astype(np.int64) ** 2).sum()), 1).reshape(-1), d.uniform(int((ns.astype(np.int64) * nrhs).sum()), 1).reshape(-1)
    eye = torch.eye(int(ns.max()), dtype=F64, device="cuda")
    at = bt = 0
    for i in range(len(ns)):
        n, r = int(ns[i]), int(nrhs[i])
        M = a[at:at + n * n].reshape(n, n)
        if kinds[i] == 0:
            torch.add(M, eye[:n, :n], alpha=float(n), out=a_view(i))
        else:
            torch.addmm(eye[:n, :n], M, M.t(), alpha=1.0 / n, out=a_view(i))
        b_view(i).copy_(b[bt:bt + n * r].reshape(r, n).t())
        at, bt = at + n * n, bt + n * r


class _MixedContext:
    """The workspace handle that a program with its own streams keeps."""

    def __init__(self):
        self.L, self.h = _lib.load(), ctypes.c_void_p()
        if self.L.bola_mixed_ctx_create(ctypes.byref(self.h)) != 0:
            raise RuntimeError(self.L.bola_last_error().decode())

    def __del__(self):
        if self.h:
            self.L.bola_mixed_ctx_destroy(self.h)
            self.h = ctypes.c_void_p()


def prepare(case, seed):
    s, op = {"case": case}, case["op"]
    x = _inputs(case, seed)
    if op == "batch":
        batch = Batch(x["ns"], x["nrhs"], x["kinds"])
        _fill(x["ns"], x["nrhs"], x["kinds"], x["draw"], batch.a_view, batch.b_view)
        s.update(batch=batch, a0=batch.A.clone(), b0=batch.B.clone())
        return s
    for key, M in x.items():
        s[key + "0"] = _flat(M)
        s[key] = s[key + "0"].clone()
    if op == "lu":
        s["ipiv"] = torch.zeros(case["n"], dtype=torch.int32, device="cuda")
    if op == "mixed":
        s.update(ctx=_MixedContext(), x=torch.zeros_like(s["b"]), info=_lib.MixedInfo(),
                 opts=_lib.MixedOpts(case["kind"], 30, 1e-14, 1, 1, 1))
    return s


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        if case["beta"] != 0.0:
            s["c"].copy_(s["c0"])
        api.gemm(case["ta"], case["tb"], m, n, k, case["alpha"], s["a"], m if case["ta"] == "N" else k,
                 s["b"], k if case["tb"] == "N" else n, case["beta"], s["c"], m)
        return s["c"]
    if op == "syrk":
        n, k = case["n"], case["k"]
        s["c"].copy_(s["c0"])
        api.syrk(case["uplo"], case["trans"], n, k, case["alpha"], s["a"], n if case["trans"] == "N" else k, case["beta"], s["c"], n)
        return s["c"]
    if op == "lu":
        m, n = case["m"], case["n"]
        s["a"].copy_(s["a0"])
        api.getrf(m, n, s["a"], m, s["ipiv"])
        out = {"lu": s["a"], "ipiv": s["ipiv"]}
        if case["nrhs"]:
            s["b"].copy_(s["b0"])
            api.getrs(n, case["nrhs"], s["a"], n, s["ipiv"], s["b"], n)
            out["x"] = s["b"]
        return out
    if op == "chol":
        n = case["n"]
        s["a"].copy_(s["a0"])
        api.potrf(case["uplo"], n, s["a"], n)
        out = {"factor": s["a"]}
        if case["nrhs"]:
            s["b"].copy_(s["b0"])
            api.potrs(case["uplo"], n, case["nrhs"], s["a"], n, s["b"], n)
            out["x"] = s["b"]
        return out
    if op == "trsm":
        m, n = case["m"], case["n"]
        s["b"].copy_(s["b0"])
        api.trsm(case["side"], case["uplo"], case["ta"], case["diag"], m, n, case["alpha"], s["a"],
                 m if case["side"] == "L" else n, s["b"], m)
        return s["b"]
    if op == "mixed":
        n, L = case["n"], s["ctx"].L
        solve = L.bola_dposv_mixed_ctx if case["spd"] else L.bola_dgesv_mixed_ctx
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        st = solve(s["ctx"].h, n, case["nrhs"], _ptr(s["a"]), n, _ptr(s["b"]), n, _ptr(s["x"]), n, ctypes.byref(s["opts"]),
                   ctypes.byref(s["info"]), stream)
        if st != 0 or s["info"].backward_error > 1e-14:
            raise RuntimeError(f"status {st}, backward error {s['info'].backward_error}: {L.bola_last_error().decode()}")
        return s["x"]
    batch = s["batch"]
    batch.A.copy_(s["a0"])
    batch.B.copy_(s["b0"])
    batch.solve(graph=case["graph"])
    return {"factors": batch.A, "x": batch.B, "info": batch.info}


def work(case):
    op = case["op"]
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * k + k * n + m * n * (2 if case["beta"] != 0.0 else 1)), "flops": 2 * m * n * k}
    if op == "syrk":
        n, k = case["n"], case["k"]
        return {"bytes": 8 * (n * k + n * (n + 1)), "flops": n * (n + 1) * k}
    if op == "lu":
        m, n, r = case["m"], case["n"], case["nrhs"]
        return {"bytes": 8 * (2 * m * n + 2 * n * r) + 4 * n, "flops": m * n * n - n ** 3 / 3 + 2 * n * n * r}
    if op == "chol":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8 * (n * (n + 1) + 2 * n * r), "flops": n ** 3 / 3 + 2 * n * n * r}
    if op == "trsm":
        m, n = case["m"], case["n"]
        t = m if case["side"] == "L" else n
        return {"bytes": 8 * (t * (t + 1) // 2 + 2 * m * n), "flops": t * m * n}
    if op == "mixed":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8 * (n * n + 2 * n * r), "flops": (1 if case["spd"] else 2) * n ** 3 / 3 + 2 * n * n * r}
    ns, nrhs, kinds = _sizes(case)
    n, r = ns.astype(np.float64), nrhs.astype(np.float64)
    return {"bytes": float((8 * (2 * n * n + 2 * n * r)).sum()), "flops": float((n ** 3 * (2 - kinds) / 3 + 2 * n * n * r).sum())}


# ---- what torch gives in 64 bits -----------------------------------------------

def exact(case, seed):
    op, x = case["op"], _inputs(case, seed)
    if op == "gemm":
        a = x["a"] if case["ta"] == "N" else x["a"].t()
        b = x["b"] if case["tb"] == "N" else x["b"].t()
        return _flat(case["alpha"] * (a @ b) + case["beta"] * x["c"])
    if op == "syrk":
        a = x["a"] if case["trans"] == "N" else x["a"].t()
        full = case["alpha"] * (a @ a.t()) + case["beta"] * x["c"]
        return _flat(torch.tril(full) + torch.triu(x["c"], 1) if case["uplo"] == "L" else torch.triu(full) + torch.tril(x["c"], -1))
    if op == "lu":
        lu, piv = torch.linalg.lu_factor(x["a"])
        out = {"lu": _flat(lu), "ipiv": None}
        if case["nrhs"]:
            out["x"] = _flat(torch.linalg.lu_solve(lu, piv, x["b"]))
        return out
    if op == "chol":
        f = torch.linalg.cholesky(x["a"])
        out = {"factor": _flat(f + torch.triu(x["a"], 1) if case["uplo"] == "L" else f.t() + torch.tril(x["a"], -1))}
        if case["nrhs"]:
            out["x"] = _flat(torch.cholesky_solve(x["b"], f))
        return out
    if op == "trsm":
        a = x["a"] if case["ta"] == "N" else x["a"].t()
        upper = (case["uplo"] == "U") == (case["ta"] == "N")
        return _flat(torch.linalg.solve_triangular(a, case["alpha"] * x["b"], upper=upper, left=case["side"] == "L",
                                                   unitriangular=case["diag"] == "U"))
    if op == "mixed":
        # one step of refinement, so that the direct solve's own error stays below what is compared
        lu, piv = torch.linalg.lu_factor(x["a"])
        y = torch.linalg.lu_solve(lu, piv, x["b"])
        return _flat(y + torch.linalg.lu_solve(lu, piv, x["b"] - x["a"] @ y))
    ns, nrhs, kinds = x["ns"], x["nrhs"], x["kinds"]
    am = [torch.empty(int(n), int(n), dtype=F64, device="cuda") for n in ns]
    bm = [torch.empty(int(n), int(r), dtype=F64, device="cuda") for n, r in zip(ns, nrhs)]
    _fill(ns, nrhs, kinds, x["draw"], am.__getitem__, bm.__getitem__)
    sol = [torch.linalg.solve(a, b) for a, b in zip(am, bm)]
    return {"factors": None, "x": torch.cat([_flat(v) for v in sol]), "info": None}
