"""Batched solves with row interchanges at every column, at the sizes where a
panel, a block of the triangular solves or a group's warps end: general
matrices (LU) and SPD ones, more right-hand sides than threads, a NaN column,
and systems that stop half-way.

Bounds: partial pivoting keeps |L| <= 1 up to the rounding of a reciprocal and
a product (two of 2^-53); the backward error of a solve is below 3 n 2^-53
times the growth of the factors, which stays under 16 for these sizes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 16, 17, 31, 32, 33, 48, 63, 64, 65, 97, 127, 128, 129, 193, 255, 256]


def run(systems, tuning=None):
    from bola_gb300.batch import Batch
    b = Batch([a.shape[0] for a, _, _ in systems], [r.shape[1] for _, r, _ in systems],
              [k for _, _, k in systems], tuning=tuning)
    for i, (a, r, _) in enumerate(systems):
        b.a_view(i).copy_(torch.from_numpy(a))
        b.b_view(i).copy_(torch.from_numpy(r))
    b.solve()
    torch.cuda.synchronize()
    return b


@pytest.mark.parametrize("width", [8, 12, 16])
def test_interchanges_and_edges(width):
    from bola_gb300.batch import Tuning
    rng = np.random.default_rng(width)
    systems = []
    for n in SIZES:
        a = rng.uniform(-1.0, 1.0, (n, n))
        systems.append((a, rng.uniform(-1.0, 1.0, (n, 1 + n % 5)), 0))
        systems.append((a @ a.T / n + np.eye(n), rng.uniform(-1.0, 1.0, (n, 300 if n == 33 else 3)), 1))
    b = run(systems, Tuning(panel_width=[width] * 8))
    assert int(b.info.abs().sum()) == 0
    for i, (a, r, kind) in enumerate(systems):
        n = a.shape[0]
        x = b.b_view(i).cpu().numpy()
        berr = np.abs(r - a @ x).max(0) / (np.abs(a).sum(1).max() * np.abs(x).max(0) + np.abs(r).max(0))
        assert berr.max() <= 16 * 3 * n * 2.0**-53, (n, kind, berr.max())
        if kind == 0:
            low = np.tril(b.a_view(i).cpu().numpy(), -1)
            assert np.abs(low).max(initial=0.0) <= 1.0 + 2.0**-51, n


@pytest.mark.parametrize("n,k", [(9, 0), (40, 7), (40, 8), (130, 129), (256, 100)])
def test_stops_at_the_same_column(n, k):
    """A column (LU) or pivot (Cholesky) that cannot be used ends that system
    only, at its column."""
    rng = np.random.default_rng(n + k)
    a = rng.uniform(-1.0, 1.0, (n, n))
    dead = a.copy()
    dead[:, k] = 0.0
    spd = a @ a.T / n + np.eye(n)
    bad = spd.copy()
    bad[k, k] = -1.0
    r = rng.uniform(-1.0, 1.0, (n, 2))
    b = run([(dead, r, 0), (bad, r, 1), (a, r, 0), (spd, r, 1)])
    assert b.info.cpu().tolist() == [k + 1, k + 1, 0, 0]
    nan = a.copy()
    nan[k % 3, :] = np.nan  # a NaN never wins a pivot search while a number is left
    b = run([(nan, r, 0), (a, r, 0)])
    assert int(b.info[1]) == 0 and np.isnan(b.b_view(0).cpu().numpy()).all()
