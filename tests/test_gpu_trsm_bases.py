"""The base cases of the triangular solves on both sides of every line at which
another kernel takes them: bit for bit the oracle's, in orders from 1 to 64, for
few systems and many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VARIANTS = [("L", "U", "T"), ("L", "L", "T"), ("R", "U", "N"), ("R", "L", "T"), ("R", "L", "N"), ("R", "U", "T")]
# (order, numbers of systems): 608 | 1064 descending; 912 and estimates ascending, the thread's in rounds of 128 on every
# SM (19,456); 100 n and 155 n above 32
SIZES = [(1, (3, 1000)), (5, (607, 608, 609, 913)), (8, (608, 609, 912, 913, 3001)), (9, (912, 913, 2100, 2801)),
         (16, (911, 1064, 1065, 4000, 5601, 7001)), (28, (913, 8001, 15401)), (31, (11001, 19456, 19457)),
         (32, (12000, 14001, 19456, 19457, 27001)), (33, (1065, 3300, 3301, 5115, 5116)),
         (64, (1064, 1065, 6400, 6401, 9920, 9921))]


@pytest.mark.parametrize("n,counts", SIZES, ids=[str(n) for n, _ in SIZES])
@pytest.mark.parametrize("side,uplo,trans", VARIANTS, ids=["".join(v) for v in VARIANTS])
def test_both_sides_of_each_line(oracle_lib, side, uplo, trans, n, counts):
    from gpu_backend import GpuBackend
    gpu = GpuBackend()
    rng = np.random.default_rng(n)
    a = np.asfortranarray(rng.uniform(-1.0, 1.0, (n, n)) / n + np.diag(rng.uniform(1.0, 2.0, n)))
    a[n // 2, n // 3] = a[n // 3, n // 2] = 0.0 if n > 2 else a[0, 0]  # BOLA skips a zero coefficient on the right
    for systems in counts:
        m, k = (n, systems) if side == "L" else (systems, n)
        b = np.asfortranarray(rng.uniform(-1.0, 1.0, (m, k)))
        for diag in "NU":
            want, got = b.copy(order="F"), b.copy(order="F")
            oracle_lib.trsm(side, uplo, trans, diag, m, k, 0.75, a, n, want, m)
            gpu.trsm(side, uplo, trans, diag, m, k, 0.75, a, n, got, m)
            assert np.array_equal(got, want), (diag, systems)
