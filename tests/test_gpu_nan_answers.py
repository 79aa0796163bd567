"""A NaN in a system is never reported as solved: the backward error is infinite,
whether the NaN stands in the matrix, in a right-hand side, or came into x."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def system(n, spd, where):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    a = torch.rand(n, n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    a = a @ a.t() / n + torch.eye(n, dtype=torch.float64, device="cuda") if spd else a + n * torch.eye(
        n, dtype=torch.float64, device="cuda")
    b = torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=g)
    if where == "matrix":
        a[n // 2, n // 3] = a[n // 3, n // 2] = math.nan
    elif where == "row":
        a[n // 2, :] = a[:, n // 2] = math.nan
    elif where == "rhs":
        b[n // 2, 1] = math.nan
    else:
        b[:, 2] = math.nan
    return a, b


@pytest.mark.parametrize("where", ["matrix", "row", "rhs", "column"])
@pytest.mark.parametrize("spd", [False, True])
@pytest.mark.parametrize("kind", [2, 3])
def test_mixed_solvers(kind, spd, where):
    from bola_gb300 import _lib
    L = _lib.load()

    def P(t):
        return ctypes.c_void_p(t.data_ptr())

    n = 200
    a, b = system(n, spd, where)
    fa, fb = a.t().contiguous().reshape(-1), b.t().contiguous().reshape(-1)
    x = torch.zeros_like(fb)
    opts, info = _lib.MixedOpts(kind, 30, 1e-14, 1, 1, 1), _lib.MixedInfo()
    solve = L.bola_dposv_mixed if spd else L.bola_dgesv_mixed
    assert solve(n, 3, P(fa), n, P(fb), n, P(x), n, ctypes.byref(opts), ctypes.byref(info),
                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, L.bola_last_error()
    assert info.backward_error == math.inf


@pytest.mark.parametrize("where", ["matrix", "row", "rhs", "column"])
@pytest.mark.parametrize("n", [20, 200])
@pytest.mark.parametrize("mode", ["mixed", "fp64"])
def test_server(mode, n, where):
    from bola_gb300.serve import Server
    a, b = (t.cpu() for t in system(n, False, where))
    fa, fb = a.t().contiguous().reshape(-1), b.t().contiguous().reshape(-1)
    with Server(slots=1, small_n=64, mode=mode) as srv:
        rid = srv.submit_raw(n, 3, 0, fa.data_ptr(), fb.data_ptr())
        _, rec = srv.wait(rid, want_x=True)
        assert rec["status"] != 0 or rec["backward_error"] == math.inf, rec
