"""Conversion of A for the mixed solve: 64-column blocks whose magnitudes lie
far apart (each is scaled by a power of two of its own), entries that leave
FP32's normal range after the scaling, zeros of both signs, and sizes with a
ragged last block.  The solve still has to reach the solver's own backward
error target."""
import numpy as np
import pytest
import torch

from test_gpu_mixed import berr, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("n", [65, 130, 257])
def test_blocks_of_different_magnitude(kind, n):
    rng = np.random.default_rng(n)
    A = rng.uniform(-1.0, 1.0, (n, n)) + 2.0 * np.sqrt(n) * np.eye(n)
    A[rng.random((n, n)) < 0.1] *= 2.0**-135  # subnormal as FP32, and below
    A[rng.random((n, n)) < 0.1] *= 0.0
    np.fill_diagonal(A, 2.0 * np.sqrt(n))
    A *= np.exp2(np.array([0, 30, -20, 10, -30])[np.arange(n) // 64])
    b = A @ rng.uniform(-1.0, 1.0, (n, 2))
    At = torch.from_numpy(A.ravel(order="F").copy()).cuda()
    bt = torch.from_numpy(b.ravel(order="F").copy()).cuda()
    x, info = solve(At, bt, n, 2, kind, fallback=0)
    assert info.backward_error <= 1e-14
    assert berr(At, x, bt, n, 2) <= 1e-14
