"""A captured factorisation as a graph like any other: cloned, nested in another
graph, instantiated twice, replayed from each form with the bits of the direct
call; the memory that it uses comes back when the forms are gone."""
import ctypes

import numpy as np
import pytest
import torch

from bola_gb300 import _lib
from bola_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


class Driver:
    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")

    def __getattr__(self, name):
        f = getattr(self.cu, name)

        def call(*args):
            r = f(*args)
            assert r == 0, (name, r)
        return call


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def capture(d, stream, m, n, a, piv, info):
    L, g = _lib.load(), ctypes.c_void_p()
    s = ctypes.c_void_p(stream.cuda_stream)
    d.cuStreamBeginCapture_v2(s, 0)  # (the strictest mode)
    st = L.bola_dgetrf(m, n, _p(a), m, _p(piv), _p(info), s)
    d.cuStreamEndCapture(s, ctypes.byref(g))
    assert st == 0, L.bola_last_error()
    return g


@pytest.mark.parametrize("m,n", [(33, 33), (200, 150), (300, 700), (600, 600)])
def test_forms_of_a_captured_factorisation(m, n):
    d, L = Driver(), _lib.load()
    a0 = torch.from_numpy(wl.uniform_matrix(m, n, seed=m, lo=-1, hi=1).ravel(order="F").copy()).cuda()
    a, piv = a0.clone(), torch.zeros(min(m, n), dtype=torch.int32, device="cuda")
    info = torch.ones(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    s = ctypes.c_void_p(stream.cuda_stream)
    torch.cuda.synchronize()
    assert L.bola_dgetrf(m, n, _p(a), m, _p(piv), _p(info), s) == 0
    torch.cuda.synchronize()
    want, wpiv = a.clone(), piv.clone()
    g = capture(d, stream, m, n, a, piv, info)
    execs, graphs = [], [g]
    clone, outer, node = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    d.cuGraphClone(ctypes.byref(clone), g)
    d.cuGraphCreate(ctypes.byref(outer), 0)
    d.cuGraphAddChildGraphNode(ctypes.byref(node), outer, None, ctypes.c_size_t(0), g)
    graphs += [clone, outer]
    for src in (g, g, clone, outer):
        execs.append(ctypes.c_void_p())
        d.cuGraphInstantiateWithFlags(ctypes.byref(execs[-1]), src, ctypes.c_ulonglong(0))
    for x in graphs:  # (the executables keep what they need)
        d.cuGraphDestroy(x)
    for x in execs:
        a.copy_(a0)
        piv.zero_()
        info.fill_(7)
        torch.cuda.synchronize()
        d.cuGraphLaunch(x, s)
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(piv, wpiv) and int(info[0]) == 0
    for x in execs:
        d.cuGraphExecDestroy(x)


def test_memory_of_graphs_comes_back():
    d, L = Driver(), _lib.load()
    n = 400
    a = torch.rand(n * n, dtype=torch.float64, device="cuda")
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    assert L.bola_dgetrf(n, n, _p(a), n, _p(piv), _p(info), ctypes.c_void_p(stream.cuda_stream)) == 0
    torch.cuda.synchronize()
    free = []
    for round_ in range(8):
        graphs = [capture(d, stream, n, n, a, piv, info) for _ in range(40)]  # 40 blocks in use at a time
        for g in graphs:
            d.cuGraphDestroy(g)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] <= 8 << 20, free


def test_direct_calls_beside_a_capture():
    """While one stream is being captured, a call on another runs at once, and neither disturbs the other (a captured
    call's streams stay part of the capture until it ends)."""
    d, L = Driver(), _lib.load()
    n = 600
    a0 = torch.from_numpy(wl.uniform_matrix(n, n, seed=9, lo=-1, hi=1).ravel(order="F").copy()).cuda()
    s0 = torch.from_numpy(wl.spd_matrix(n, seed=9).ravel(order="F").copy()).cuda()
    bufs = [(a0.clone(), s0.clone(), torch.zeros(n, dtype=torch.int32, device="cuda"),
             torch.ones(2, dtype=torch.int32, device="cuda")) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()

    def calls(stream, a, sp, piv, info):
        s = ctypes.c_void_p(stream.cuda_stream)
        assert L.bola_dgetrf(n, n, _p(a), n, _p(piv), _p(info), s) == 0, L.bola_last_error()
        assert L.bola_dpotrf(b"L", n, _p(sp), n, _p(info[1:]), s) == 0, L.bola_last_error()

    calls(streams[1], *bufs[1])  # (attributes, pools)
    torch.cuda.synchronize()
    want = [t.clone() for t in bufs[1]]
    g, x = ctypes.c_void_p(), ctypes.c_void_p()
    s = ctypes.c_void_p(streams[0].cuda_stream)
    d.cuStreamBeginCapture_v2(s, 2)  # (relaxed: other streams' calls are allowed)
    calls(streams[0], *bufs[0])
    bufs[1][0].copy_(a0)
    bufs[1][1].copy_(s0)
    torch.cuda.default_stream().synchronize()
    calls(streams[1], *bufs[1])
    calls_again = [t.clone() for t in (a0, s0)] + [torch.zeros_like(want[2]), torch.ones_like(want[3])]
    torch.cuda.default_stream().synchronize()
    calls(streams[1], *calls_again)
    d.cuStreamEndCapture(s, ctypes.byref(g))
    torch.cuda.synchronize()
    for got in (bufs[1], calls_again):
        assert all(torch.equal(t, w) for t, w in zip(got, want))
    d.cuGraphInstantiateWithFlags(ctypes.byref(x), g, ctypes.c_ulonglong(0))
    d.cuGraphLaunch(x, s)
    torch.cuda.synchronize()
    assert all(torch.equal(t, w) for t, w in zip(bufs[0], want))
    d.cuGraphExecDestroy(x)
    d.cuGraphDestroy(g)
