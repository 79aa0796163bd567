"""Cholesky blocks that stop, at every column of a block: the warps that share
a block agree on the column, in a run of many launches (a warp that saw the
stop one column early would leave the others waiting), and what they leave is
the oracle's state."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def indefinite(n, k, seed):
    """SPD but for the pivot of column k (0-based), which is negative."""
    rng = np.random.default_rng(seed)
    h = rng.uniform(-1.0, 1.0, (n, n))
    a = np.asfortranarray(h @ h.T / n + np.eye(n))
    a[k, k] = -1.0
    return a


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n", [1, 7, 31, 32])
def test_every_column_of_a_block(oracle_lib, uplo, n):
    from bola_gb300 import _lib
    L = _lib.load()
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    for k in range(n):
        a = indefinite(n, k, 100 * n + k)
        want = a.copy(order="F")
        assert oracle_lib.potrf(uplo, n, want, n) == k + 1
        a0 = torch.from_numpy(a.ravel(order="F").copy()).cuda()
        t = torch.empty_like(a0)
        for _ in range(8):
            t.copy_(a0)
            assert L.bola_dpotrf(uplo.encode(), n, ctypes.c_void_p(t.data_ptr()), n, ctypes.c_void_p(info.data_ptr()),
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            assert int(info[0]) == k + 1
            assert np.array_equal(t.cpu().numpy().reshape(n, n, order="F"), want)


@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("n", [64, 150])
def test_every_column_of_the_mixed_factor(kind, n):
    """The FP32 and the FP64 block; the mixed LU then takes the system over."""
    from bola_gb300 import _lib
    L = _lib.load()

    def P(t):
        return ctypes.c_void_p(t.data_ptr())

    ctx = ctypes.c_void_p()
    assert L.bola_mixed_ctx_create(ctypes.byref(ctx)) == 0
    for k in range(n):
        a = torch.from_numpy(indefinite(n, k, k)).cuda()
        b = torch.ones(n, dtype=torch.float64, device="cuda")
        x = torch.zeros_like(b)
        flat = a.t().contiguous().reshape(-1)
        opts, info = _lib.MixedOpts(kind, 30, 1e-14, 0, 1, 0), _lib.MixedInfo()
        st = L.bola_dposv_mixed_ctx(ctx, n, 1, P(flat), n, P(b), n, P(x), n, ctypes.byref(opts), ctypes.byref(info),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0, L.bola_last_error()
        assert info.factor_info == k + 1 and info.factorization == 0 and info.backward_error <= 1e-14
    L.bola_mixed_ctx_destroy(ctx)
