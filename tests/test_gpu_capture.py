"""The FP64 calls recorded into a CUDA graph (programmatic dependents, forks
onto the library's streams and all) and replayed: the bits of direct calls."""
import ctypes

import numpy as np
import pytest
import torch

from bola_gb300 import _lib
from bola_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _calls(n, A, S, B, C, piv, info):
    L = _lib.load()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    u, lo, t, nt = (ctypes.c_char(c) for c in (b"U", b"L", b"T", b"N"))
    f = ctypes.c_double
    assert L.bola_dgemm(nt, t, n, n, 70, f(-1.0), _p(B), n, _p(B), n, f(1.0), _p(C), n, s) == 0
    assert L.bola_dgetrf(n, n, _p(A), n, _p(piv), _p(info), s) == 0
    assert L.bola_dtrsm(lo, lo, nt, u, n, 90, f(1.0), _p(A), n, _p(B), n, s) == 0
    assert L.bola_dpotrf(u, n, _p(S), n, _p(info[1:]), s) == 0


@pytest.mark.parametrize("n", [200, 600])
def test_graph_replays_the_same_bits(n):
    A0 = wl.uniform_matrix(n, n, seed=n, lo=-1, hi=1)
    S0 = A0 @ A0.T / n + np.eye(n)
    host = [A0, S0, wl.uniform_matrix(n, 90, seed=1, lo=-1, hi=1), wl.uniform_matrix(n, n, seed=2, lo=-1, hi=1)]
    orig = [torch.from_numpy(np.asfortranarray(x).ravel(order="F").copy()).cuda() for x in host]
    bufs = [t.clone() for t in orig]
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(2, dtype=torch.int32, device="cuda")
    _calls(n, *bufs, piv, info)  # (also sets up streams, attributes and pools)
    torch.cuda.synchronize()
    want, wpiv = [t.clone() for t in bufs], piv.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        _calls(n, *bufs, piv, info)
    for _ in range(2):
        for b, o in zip(bufs, orig):
            b.copy_(o)
        piv.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert int(info.abs().sum()) == 0
        assert torch.equal(piv, wpiv)
        for b, w in zip(bufs, want):
            assert torch.equal(b, w)
