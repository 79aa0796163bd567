"""The FP64 kernels against the oracle, bit for bit, where their forms change
over: every tile plan of the product (64x64, 32x32 with 16x16, 8x8, K split
over a cluster and over memory, block triangles) with ragged edges, the base
cases of the triangular solve by number of systems, the diagonal blocks of
SYRK by number of blocks, and the Cholesky around its block sizes."""
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


def same(a, b):
    return np.array_equal(a, b, equal_nan=True)


GEMM = [(1235, 1093, 64), (1235, 1093, 130),              # 64x64 cells, with and without a remainder of 16x16
        (700, 301, 90), (333, 260, 33),                   # 32x32 and 16x16
        (41, 38, 64), (8, 4, 1),                          # 8x8
        (64, 64, 1000), (97, 66, 513), (130, 40, 129),    # K over clusters
        (256, 256, 4096), (260, 131, 2050),               # K over memory
        (7, 900, 65), (900, 3, 65)]                       # edges only


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("alpha,beta", [(1.0, 1.0), (-0.5, 0.0)])
def test_gemm_plans(both, ta, tb, alpha, beta):
    g, o = both
    for m, n, k in GEMM:
        A = wl.uniform_matrix(*((m, k) if ta == "N" else (k, m)), seed=m, lo=-1, hi=1)
        B = wl.uniform_matrix(*((k, n) if tb == "N" else (n, k)), seed=n, lo=-1, hi=1)
        C = wl.uniform_matrix(m, n, seed=k, lo=-1, hi=1)
        C1, C2 = C.copy(order="F"), C.copy(order="F")
        o.gemm(ta, tb, m, n, k, alpha, A, A.shape[0], B, B.shape[0], beta, C1, m)
        g.gemm(ta, tb, m, n, k, alpha, A, A.shape[0], B, B.shape[0], beta, C2, m)
        assert same(C1, C2), (m, n, k)


@pytest.mark.parametrize("uplo,trans", [("L", "N"), ("U", "T")])
def test_syrk_blocks(both, uplo, trans):
    g, o = both
    for n in [1, 17, 31, 32, 33, 63, 479, 481, 512, 545, 1300]:
        for k in [1, 32, 33, 70] if n < 1000 else [70]:
            A = wl.uniform_matrix(*((n, k) if trans == "N" else (k, n)), seed=n + k, lo=-1, hi=1)
            A[n // 3 % A.shape[0], k // 2 % A.shape[1]] = 0.0  # BOLA skips a zero multiplier
            C = wl.uniform_matrix(n, n, seed=k, lo=-1, hi=1)
            C1, C2 = C.copy(order="F"), C.copy(order="F")
            o.syrk(uplo, trans, n, k, -1.0, A, A.shape[0], 1.0, C1, n)
            g.syrk(uplo, trans, n, k, -1.0, A, A.shape[0], 1.0, C2, n)
            assert same(C1, C2), (n, k)


@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("diag", ["N", "U"])
def test_trsm_bases(both, side, uplo, ta, diag):
    g, o = both
    for k, systems in [(32, 912), (32, 913), (19, 1001), (1, 1300), (33, 1216), (64, 1217), (47, 8195)]:
        m, n = (k, systems) if side == "L" else (systems, k)
        A = wl.uniform_matrix(k, k, seed=k, lo=-1, hi=1)
        A[np.diag_indices(k)] += np.sqrt(k) + 1.0
        B = wl.uniform_matrix(m, n, seed=8, lo=-1, hi=1)
        B1, B2 = B.copy(order="F"), B.copy(order="F")
        o.trsm(side, uplo, ta, diag, m, n, 1.5, A, k, B1, m)
        g.trsm(side, uplo, ta, diag, m, n, 1.5, A, k, B2, m)
        assert same(B1, B2), (m, n)


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 319, 320, 321, 351, 640, 653])
def test_potrf_blocks(both, uplo, n):
    g, o = both
    A = wl.uniform_matrix(n, n, seed=n, lo=-1, hi=1)
    A = np.asfortranarray(A @ A.T / n + np.eye(n))
    A1, A2 = A.copy(order="F"), A.copy(order="F")
    assert o.potrf(uplo, n, A1, n) == 0
    assert g.potrf(uplo, n, A2, n) == 0
    assert same(A1, A2)


@pytest.mark.parametrize("n,nrhs", [(32, 3), (33, 1), (200, 3), (257, 300), (1025, 5), (3100, 2)])
def test_getrs_rows(both, n, nrhs):
    """Interchanges that move rows anywhere (not only down), the solve after them."""
    g, o = both
    rng = np.random.default_rng(n)
    A = wl.uniform_matrix(n, n, seed=n, lo=-1, hi=1) / n
    A[np.diag_indices(n)] = 2.0 + rng.random(n)
    piv = rng.integers(1, n + 1, n).astype(np.int32)
    piv[::3] = np.arange(1, n + 1)[::3]
    B = wl.uniform_matrix(n + 3, nrhs, seed=2, lo=-1, hi=1)
    B1, B2 = B.copy(order="F"), B.copy(order="F")
    o.laswp(nrhs, B1, n + 3, 1, n, piv, 1)
    o.trsm("L", "L", "N", "U", n, nrhs, 1.0, A, n, B1, n + 3)
    o.trsm("L", "U", "N", "N", n, nrhs, 1.0, A, n, B1, n + 3)
    g.getrs(n, nrhs, A, n, piv, B2, n + 3)
    assert same(B1, B2)
