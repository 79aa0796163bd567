"""DGEMM with small outputs and a deep K, where K is split over the GPU: bit for
bit the oracle's, with and without memory for the partial sums, at the numbers
of 64-deep chunks where a split's parts, passes and the fold's batches end, and
with partial sums beyond what the scratch pool keeps."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def both(m, n, k, beta, seed, names, oracle_lib, ta="N", tb="N"):
    from bola_gb300 import _lib
    L = _lib.load()
    rng = np.random.default_rng(seed)
    a = np.asfortranarray(rng.uniform(-1.0, 1.0, (m, k) if ta == "N" else (k, m)))
    b = np.asfortranarray(rng.uniform(-1.0, 1.0, (k, n) if tb == "N" else (n, k)))
    c = np.asfortranarray(rng.uniform(-1.0, 1.0, (m, n)))
    want = c.copy(order="F")
    oracle_lib.gemm(ta, tb, m, n, k, -0.75, a, a.shape[0], b, b.shape[0], beta, want, m)
    ga, gb, gc = (torch.from_numpy(x.ravel(order="F")).cuda() for x in (a, b, c))
    for name in names:
        t = gc.clone()
        st = getattr(L, name)(ta.encode(), tb.encode(), m, n, k, -0.75, ctypes.c_void_p(ga.data_ptr()), a.shape[0],
                              ctypes.c_void_p(gb.data_ptr()), b.shape[0], beta, ctypes.c_void_p(t.data_ptr()), m,
                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0, L.bola_last_error()
        assert np.array_equal(t.cpu().numpy().reshape(m, n, order="F"), want), (name, m, n, k)


@pytest.mark.parametrize("m,n", [(8, 4), (13, 9), (16, 16), (40, 28), (64, 64), (100, 33), (128, 128)])
@pytest.mark.parametrize("chunks", [9, 15, 16, 17, 32, 33, 64, 65, 127, 129, 300])
def test_chunks_of_a_split(oracle_lib, m, n, chunks):
    for k in (64 * chunks - 1, 64 * chunks, 64 * chunks - 55):
        both(m, n, k, 0.5, m + k, ("bola_dgemm", "bola_dgemm_noalloc"), oracle_lib)


@pytest.mark.parametrize("ta,tb", [("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", [(21, 18, 2501), (64, 64, 5000), (70, 65, 4097)])
def test_transposed_operands(oracle_lib, ta, tb, m, n, k):
    both(m, n, k, 1.0, k, ("bola_dgemm", "bola_dgemm_noalloc"), oracle_lib, ta, tb)


@pytest.mark.parametrize("m,n,k", [(64, 64, 140_000), (128, 128, 34_000), (16, 16, 300_000)])
def test_very_deep(oracle_lib, m, n, k):
    both(m, n, k, 1.0, k, ("bola_dgemm",), oracle_lib)


def test_the_limit_without_memory():
    """64 x 64: a chunk's partial sums are 32 KiB, so 2048 chunks (64 MiB) are taken, more are not up to 32,768 (1 GiB),
    and a refused call leaves C alone."""
    from bola_gb300 import _lib
    L = _lib.load()
    m = n = 64
    k = 64 * 32768 + 1
    a = torch.rand(m * k, dtype=torch.float64, device="cuda")
    c0 = torch.rand(m * n, dtype=torch.float64, device="cuda")
    for depth, status in [(64 * 2048, 0), (64 * 2048 + 1, -1002), (64 * 32768, -1002), (64 * 32768 + 1, 0)]:
        c = c0.clone()
        st = L.bola_dgemm_noalloc(b"N", b"T", m, n, depth, 1.0, ctypes.c_void_p(a.data_ptr()), m,
                                  ctypes.c_void_p(a.data_ptr()), n, 1.0, ctypes.c_void_p(c.data_ptr()), m,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == status, (depth, st)
        torch.cuda.synchronize()
        assert torch.equal(c, c0) == (status != 0)
        if status:
            assert b"does not take shapes beyond" in L.bola_last_error()


def test_deep_product_when_memory_is_short():
    """Partial sums of a gigabyte where 0.6 GB are free: the product is formed without them, with the same bits."""
    from bola_gb300 import _lib
    L = _lib.load()
    m = n = 128
    k = 500_000

    def product(c):
        return L.bola_dgemm(b"N", b"T", m, n, k, 1.0, ctypes.c_void_p(a.data_ptr()), m, ctypes.c_void_p(b.data_ptr()), n,
                            1.0, ctypes.c_void_p(c.data_ptr()), m,
                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))

    a, b = (torch.rand(m * k, dtype=torch.float64, device="cuda") - 0.5 for _ in range(2))
    c0 = torch.rand(m * n, dtype=torch.float64, device="cuda")
    c1, c2 = c0.clone(), c0.clone()
    assert product(c1) == 0, L.bola_last_error()
    # the plan without memory, once before memory is short (its kernels are loaded then)
    warm = c0.clone()
    assert L.bola_dgemm_noalloc(b"N", b"T", m, n, 30_000, 1.0, ctypes.c_void_p(a.data_ptr()), m,
                                ctypes.c_void_p(b.data_ptr()), n, 1.0, ctypes.c_void_p(warm.data_ptr()), m,
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - 600_000_000, dtype=torch.uint8, device="cuda")
    try:
        status = product(c2)
        torch.cuda.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert status == 0, L.bola_last_error()
    assert torch.equal(c1, c2) and not torch.equal(c1, c0)
