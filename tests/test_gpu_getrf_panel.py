"""The cluster panel of getrf against the oracle, bit for bit, where its
partition of the rows can go wrong: around one CTA's 64 rows, around a row
group's 32 and a cluster's 16 CTAs, on panels narrower than 32 columns or
shorter than wide, and on inputs that make BOLA's pivot search order and its
skipped updates matter (exact ties, zeros, NaN, infinities)."""
import numpy as np
import pytest

from bola_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[2, 4], ids=["neon", "avx2"])
def both(request, oracle_lib):
    from gpu_backend import GpuBackend
    gpu = GpuBackend()
    gpu.set_lanes(request.param)
    oracle_lib.set_lanes(request.param)
    yield gpu, oracle_lib
    gpu.set_lanes(2)
    oracle_lib.set_lanes(2)


def _factor(impl, A, m, n):
    B, p = A.copy(order="F"), np.zeros(min(m, n), np.int32)
    r = impl.getrf(m, n, B, m, p)
    return B, p, (r if isinstance(r, (int, np.integer)) else None)


def _values(kind, m, n):
    u = wl.uniform_matrix(m, n, seed=31 * m + n, lo=-1, hi=1)
    if kind == "uniform":
        return u
    if kind == "ties":  # few distinct values, many zeros: ties in every search, skipped column pairs
        return np.asfortranarray(np.round(2.0 * u))
    A = u.copy(order="F")
    A[m // 3, min(3, n - 1)] = np.nan
    A[m // 2, min(7, n - 1)] = np.inf
    return A


@pytest.mark.parametrize("kind", ["uniform", "ties", "nonfinite"])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 2), (7, 5), (15, 32), (31, 17), (33, 32), (64, 32), (65, 31), (129, 32),
                                 (1023, 32), (1025, 32), (2050, 33), (4099, 32)])
def test_panel_bitwise(both, m, n, kind):
    g, o = both
    A = _values(kind, m, n)
    A1, p1, r1 = _factor(o, A, m, n)
    A2, p2, r2 = _factor(g, A, m, n)
    assert (r1 == 0) == (r2 == 0)
    assert np.array_equal(p1, p2)
    assert np.array_equal(A1, A2, equal_nan=True)
