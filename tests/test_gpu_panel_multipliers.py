"""Partial pivoting in the low-precision LU, every kind of update: no multiplier
above 1 but by what the search and two roundings leave (pivots are compared with
the five lowest of 24 significand bits dropped, less than 2^-18, and each
rounding is 2^-24), with ragged sizes, exact ties, columns that differ in size
by many powers of two, and entries of one magnitude."""
import numpy as np
import pytest
import torch

from test_gpu_tournament_panel import factor

pytestmark = pytest.mark.gpu

LMAX = 1.0 + 2.0**-17


def matrices(n, rng):
    yield rng.uniform(-1.0, 1.0, (n, n))
    yield rng.integers(-3, 4, (n, n)) + 8.0 * np.eye(n)
    yield rng.integers(-1, 2, (n, n)) * 2.0 + np.diag(rng.integers(1, 3, n) * 0.5)
    yield rng.uniform(-1.0, 1.0, (n, n)) * 2.0 ** rng.integers(-20, 20, (1, n))
    yield np.sign(rng.uniform(-1.0, 1.0, (n, n))) * (1.0 + rng.integers(0, 3, (n, n)) * 2.0**-23)


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 7, 63, 64, 65, 129, 333, 1000])
def test_multipliers_are_bounded(kind, n):
    rng = np.random.default_rng(n)
    for i, a in enumerate(matrices(n, rng)):
        w = torch.from_numpy(a.astype(np.float32).ravel(order="F").copy()).cuda()
        ipiv, info = factor(w, n, kind)
        f = w.cpu().numpy().reshape(n, n, order="F").astype(np.float64)
        assert np.all(ipiv >= np.arange(1, n + 1)) and np.all(ipiv <= n)
        if info == 0:
            assert np.abs(np.tril(f, -1)).max(initial=0.0) <= LMAX, (i, np.abs(np.tril(f, -1)).max())
        else:  # (integer entries: an exactly singular matrix is possible)
            assert i in (1, 2), (i, info)
