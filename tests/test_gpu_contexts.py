"""The library under two contexts of one device, used in turn, and under host
threads: what it keeps stays bounded, and every launch gets the shared memory
that it asks for in the context and on the thread it is made from."""
import os
import subprocess
import sys
import textwrap
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes
import numpy as np
from bola_gb300 import _lib
cu = ctypes.CDLL("libcuda.so.1")

def ok(r):
    assert r == 0, r

ok(cu.cuInit(0))
ctxs = [ctypes.c_void_p() for _ in range(2)]
for c in ctxs:
    ok(cu.cuCtxCreate_v2(ctypes.byref(c), 0, 0))

def device(a):
    a = np.ascontiguousarray(a)
    p = ctypes.c_void_p()
    ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
    ok(cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes)))
    return p

def host(p, shape):
    out = np.empty(shape)
    ok(cu.cuMemcpyDtoH_v2(out.ctypes.data_as(ctypes.c_void_p), p, ctypes.c_size_t(out.nbytes)))
    return out

L = _lib.load()
"""


def child(body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def test_scratch_stays_bounded_under_two_contexts():
    """A product whose partial sums take 32 MiB of scratch, twelve times in each of two contexts: the library keeps at
    most 64 MiB for each."""
    child("""
    m, k = 64, 65536
    rng = np.random.default_rng(1)
    a, b = rng.uniform(-1, 1, (k, m)), rng.uniform(-1, 1, (k, m))  # row-major: the columns of the m x k operands
    want = a.T @ b
    free = []
    bufs = []
    for c in ctxs:
        ok(cu.cuCtxSetCurrent(c))
        bufs.append((device(a), device(b), device(np.zeros((m, m)))))
    for turn in range(12):
        for c, (pa, pb, pc) in zip(ctxs, bufs):
            ok(cu.cuCtxSetCurrent(c))
            st = L.bola_dgemm(b"N", b"T", m, m, k, 1.0, pa, m, pb, m, 0.0, pc, m, None)
            assert st == 0, (turn, st, L.bola_last_error())
            ok(cu.cuCtxSynchronize())
            if turn in (0, 11):
                got = host(pc, (m, m)).T
                assert np.abs(got - want).max() < 1e-9
        f, t = ctypes.c_size_t(), ctypes.c_size_t()
        ok(cu.cuMemGetInfo_v2(ctypes.byref(f), ctypes.byref(t)))
        free.append(f.value)
    assert free[1] - free[-1] <= 160 << 20, [(free[1] - v) >> 20 for v in free]
    """)


def test_scratch_of_ended_contexts_is_given_back():
    """The same product in contexts that are destroyed after it, 24 one after the other: no more is kept than for the
    eight contexts that have a pool of their own."""
    child("""
    m, k = 64, 65536
    a = np.random.default_rng(2).uniform(-1, 1, (k, m))
    want = a.T @ a
    free = []
    f, t = ctypes.c_size_t(), ctypes.c_size_t()
    for turn in range(24):
        c = ctypes.c_void_p()
        ok(cu.cuCtxCreate_v2(ctypes.byref(c), 0, 0))
        pa, pc = device(a), device(np.zeros((m, m)))
        st = L.bola_dgemm(b"N", b"T", m, m, k, 1.0, pa, m, pa, m, 0.0, pc, m, None)
        assert st == 0, (turn, st, L.bola_last_error())
        ok(cu.cuCtxSynchronize())
        assert np.abs(host(pc, (m, m)).T - want).max() < 1e-9
        for p in (pa, pc):
            ok(cu.cuMemFree_v2(p))
        ok(cu.cuCtxDestroy_v2(c))
        ok(cu.cuCtxSetCurrent(ctxs[0]))
        ok(cu.cuMemGetInfo_v2(ctypes.byref(f), ctypes.byref(t)))
        free.append(f.value)
    assert free[0] - free[-1] <= 320 << 20, [(free[0] - v) >> 20 for v in free]
    """)


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("spd", [False, True])
def test_mixed_solve_in_each_context(kind, spd):
    """The solver's kernels ask for more shared memory and larger clusters than a context grants by itself."""
    child(f"""
    n, r, kind, spd = 700, 3, {kind}, {spd}
    rng = np.random.default_rng(kind)
    a = rng.uniform(-1, 1, (n, n))
    a = a @ a.T / n + np.eye(n) if spd else a + n * np.eye(n)
    x = rng.uniform(-1, 1, (r, n))
    b = x @ a.T  # row i: the right-hand side of solution i
    for c in ctxs + ctxs:
        ok(cu.cuCtxSetCurrent(c))
        pa, pb, px = device(a.T), device(b), device(np.zeros_like(b))
        h = ctypes.c_void_p()
        ok(L.bola_mixed_ctx_create(ctypes.byref(h)))
        info = _lib.MixedInfo()
        opts = _lib.MixedOpts(kind, 30, 1e-14, 0, 1, 0)
        solve = L.bola_dposv_mixed_ctx if spd else L.bola_dgesv_mixed_ctx
        st = solve(h, n, r, pa, n, pb, n, px, n, ctypes.byref(opts), ctypes.byref(info), None)
        assert st == 0, (st, L.bola_last_error())
        ok(cu.cuCtxSynchronize())
        assert info.backward_error <= 1e-14 and info.path < 2, (info.path, info.backward_error)
        assert np.abs(host(px, (r, n)) - x).max() < 1e-10
        ok(L.bola_mixed_ctx_destroy(h))
        for p in (pa, pb, px):
            ok(cu.cuMemFree_v2(p))
    """)


def test_look_ahead_in_each_context():
    """The streams that a large factorisation overlaps on belong to a context: each has its own."""
    child("""
    n = 600
    rng = np.random.default_rng(3)
    a = rng.uniform(-1, 1, (n, n))
    s = a @ a.T / n + np.eye(n)
    first = None
    for c in ctxs + ctxs:
        ok(cu.cuCtxSetCurrent(c))
        pa, ps = device(a), device(s)
        piv, info = device(np.zeros(n, np.int32)), device(np.ones(2, np.int32))
        st = L.bola_dgetrf(n, n, pa, n, piv, info, None)
        assert st == 0, (st, L.bola_last_error())
        st = L.bola_dpotrf(b"L", n, ps, n, ctypes.c_void_p(info.value + 4), None)
        assert st == 0, (st, L.bola_last_error())
        ok(cu.cuCtxSynchronize())
        got = host(pa, (n, n)).tobytes(), host(ps, (n, n)).tobytes(), host(info, (1,)).tobytes()
        assert got[2] == bytes(8)
        assert first is None or got == first
        first = got
        for p in (pa, ps, piv, info):
            ok(cu.cuMemFree_v2(p))
    """)


def test_right_solves_from_two_threads():
    """Base cases of different orders from two host threads: neither's launch loses the shared memory that the other's
    set."""
    from bola_gb300 import api
    failures, want = [], {}

    def solve(n, reps):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                a = torch.eye(n, dtype=torch.float64, device="cuda").reshape(-1) * 2.0
                b0 = torch.arange(1500 * n, dtype=torch.float64, device="cuda")
                b = b0.clone()
                for _ in range(reps):
                    b.copy_(b0)
                    api.trsm("R", "L", "N", "N", 1500, n, 1.0, a, n, b, 1500)
                want[n] = bool(torch.equal(b, b0 * 0.5))
        except Exception as e:  # (reported by the main thread)
            failures.append((n, str(e)))

    threads = [threading.Thread(target=solve, args=(n, 3000)) for n in (64, 40)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures and want == {64: True, 40: True}, (failures, want)
