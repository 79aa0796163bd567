"""The 64-column panel of the low-precision LU at the sizes where its rows
change hands: a row per thread, 256 rows per CTA aimed at, up to 16 CTAs
(beyond 4096 rows up to 512 rows each).  P W = L U in FP64 on the host, and
partial pivoting's bound on the multipliers: pivots are compared with the five
lowest of 24 significand bits dropped, so a row's value exceeds the pivot's by
less than 2^-18 of it, and two roundings of 2^-24 follow."""
import numpy as np
import pytest
import torch

from bola_gb300 import workloads as wl
from test_gpu_tournament_panel import factor

pytestmark = pytest.mark.gpu

LMAX = 1.0 + 2.0**-17
TOL = 3e-5  # 3xTF32 updates, |P W - L U| against |L| |U| sqrt(n)


@pytest.mark.parametrize("n", [64, 65, 255, 256, 257, 260, 513, 1023, 1025, 4097])
def test_panel_row_splits(n):
    A = wl.uniform_matrix(n, n, seed=n, lo=-1.0, hi=1.0)
    W = torch.from_numpy(A.astype(np.float32).ravel(order="F").copy()).cuda()
    ipiv, info = factor(W, n, 2)
    assert info == 0
    F = W.cpu().numpy().reshape(n, n, order="F").astype(np.float64)
    Lm = np.tril(F, -1)
    assert np.abs(Lm).max() <= LMAX
    Lm += np.eye(n)
    Um = np.triu(F)
    PA = A.astype(np.float32).astype(np.float64)
    for j, p in enumerate(ipiv - 1):
        if p != j:
            PA[[j, p]] = PA[[p, j]]
    res = np.abs(PA - Lm @ Um).max() / (np.abs(Um).max() * np.sqrt(n))
    assert res <= TOL, res
