"""The mixed solvers' last resort, plain FP64, on a matrix that turns out to be
singular there: no row outside the right-hand sides is named by an interchange
that was never written, and the answer is reported as what it is."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def matrix(n):
    """Unit diagonal; rows 0 and 1 nearly equal (the FP32 Cholesky gives up after its first panel), rows 130 and 131
    equal (the FP64 LU meets a zero pivot at column 132, in its fifth panel)."""
    a = torch.eye(n, dtype=torch.float64, device="cuda")
    a[0, 1] = a[1, 0] = 1.0 - 2.0**-20
    a[130, 131] = a[131, 130] = 1.0
    return a.reshape(-1)


@pytest.mark.parametrize("spd", [True, False])
def test_singular_matrix_reaches_the_fallback(spd):
    from bola_gb300 import _lib
    L = _lib.load()

    def P(t):
        return ctypes.c_void_p(t.data_ptr())

    n, r = 300, 4
    a = matrix(n)
    pad = torch.full(((r + 2) * n,), 5.0, dtype=torch.float64, device="cuda")
    x = pad[n:(r + 1) * n]
    b = torch.rand(n * r, dtype=torch.float64, device="cuda")
    ctx = ctypes.c_void_p()
    assert L.bola_mixed_ctx_create(ctypes.byref(ctx)) == 0
    opts, info = _lib.MixedOpts(2, 30, 1e-14, 1, 1, 0), _lib.MixedInfo()
    solve = L.bola_dposv_mixed_ctx if spd else L.bola_dgesv_mixed_ctx
    st = solve(ctx, n, r, P(a), n, P(b), n, P(x), n, ctypes.byref(opts), ctypes.byref(info),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert st == 0 and info.path == 2
    assert not info.backward_error <= 1e-14 or math.isnan(info.backward_error)
    assert bool((pad[:n] == 5.0).all()) and bool((pad[(r + 1) * n:] == 5.0).all())
    L.bola_mixed_ctx_destroy(ctx)
