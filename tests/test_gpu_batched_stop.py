"""What a batched LU leaves of a singular system: the state of the elimination
at the column that has no pivot, row interchanges before it included, in A and
in the right-hand sides.

The elimination of a panel of `width` columns updates the panel's columns only;
the columns after the panel have the panel's interchanges and the updates of the
panels before it.  Bounds: numpy rounds product and sum where the kernel fuses
them, so elements of size g that take up to n multiply-adds differ by n g 2^-52
at first, and the elimination carries that on times the condition of the block
eliminated; interchanges alone change no bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def stopped(a, b, width):
    """numpy's elimination in the order above; the column that stops it (1-based, or 0) and the interchanges done."""
    a, b, n, swaps = a.copy(), b.copy(), a.shape[0], 0
    for k0 in range(0, n, width):
        end = min(k0 + width, n)
        for k in range(k0, end):
            p = k + int(np.argmax(np.abs(a[k:, k])))
            if a[p, k] == 0.0:
                return a, b, k + 1, swaps
            swaps += p != k
            a[[k, p]], b[[k, p]] = a[[p, k]], b[[p, k]]
            a[k + 1:, k] *= 1.0 / a[k, k]
            a[k + 1:, k + 1:end] -= np.outer(a[k + 1:, k], a[k, k + 1:end])
        for r in range(k0, end):
            a[r, end:] -= a[r, k0:r] @ a[k0:r, end:]
        a[end:, end:] -= a[end:, k0:end] @ a[k0:end, end:]
    return a, b, 0, swaps


@pytest.mark.parametrize("width", [8, 12, 16])
@pytest.mark.parametrize("n,k", [(4, 2), (20, 12), (33, 17), (40, 7), (40, 8), (64, 63), (100, 50), (130, 129), (256, 100)])
def test_state_at_a_zero_pivot(n, k, width):
    from bola_gb300.batch import Batch, Tuning
    rng = np.random.default_rng(1000 * n + k)
    a = rng.uniform(-1.0, 1.0, (n, n))
    a[:, k] = 0.0
    b = rng.uniform(-1.0, 1.0, (n, 3))
    want_a, want_b, info, swaps = stopped(a, b, width)
    assert info == k + 1 and swaps > 0
    batch = Batch([n], [3], [0], tuning=Tuning(panel_width=[width] * 8))
    batch.a_view(0).copy_(torch.from_numpy(a))
    batch.b_view(0).copy_(torch.from_numpy(b))
    batch.solve()
    torch.cuda.synchronize()
    assert int(batch.info[0]) == info
    block = (np.tril(want_a[:k, :k], -1) + np.eye(k)) @ np.triu(want_a[:k, :k])
    bound = n * np.abs(want_a).max() * 2.0**-52 * np.linalg.cond(block)
    assert bound < 1e-6  # (rows in the wrong place are off by 0.1 and more)
    assert np.abs(batch.a_view(0).cpu().numpy() - want_a).max() <= bound
    assert np.array_equal(batch.b_view(0).cpu().numpy(), want_b)
