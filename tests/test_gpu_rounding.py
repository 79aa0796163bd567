"""The quotient, reciprocal and square root that every FP64 factor is made of,
bit for bit against IEEE arithmetic: systems of order one and two, whose solves
are nothing else (LU 1 x 1: b / a; 2 x 2: a21 (1 / a11); Cholesky 1 x 1:
sqrt(a), then b / l / l).  Values over the whole exponent range, its ends,
subnormals, infinities, and significands whose quotients and roots lie beside a
midpoint between two doubles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def same(got, want):
    return np.array_equal(got.view(np.int64), want.view(np.int64)) or bool(
        np.all((got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))))


def numbers(rng, count):
    bits = rng.integers(0, 2**52, count, dtype=np.int64)
    # significands of few bits, of all ones, and beside a power of two
    few = rng.integers(0, 2**20, count, dtype=np.int64) << 32
    ends = np.where(rng.random(count) < 0.5, 2**52 - 1 - rng.integers(0, 64, count), rng.integers(0, 64, count))
    kind = rng.integers(0, 4, count)
    mant = np.where(kind == 0, few, np.where(kind == 1, ends, bits))
    expo = np.where(rng.random(count) < 0.6, rng.integers(1003, 1043, count), rng.integers(0, 2047, count))
    special = np.array([1, 2, 2**52 - 1, 2**52, 2**52 + 1, 0x7fefffffffffffff, 0x7ff0000000000000, 1023 << 52,
                        (1023 << 52) - 1, 0x4000000000000000 - 1], dtype=np.int64)
    out = (expo.astype(np.int64) << 52) | mant
    out[:special.size] = special
    out[out == 0] = 1
    return out.view(np.float64)


def solve(ns, kinds, a, b):
    from bola_gb300.batch import Batch
    batch = Batch(ns, np.ones(len(ns), np.int32), kinds)
    batch.A.copy_(torch.from_numpy(a))
    batch.B.copy_(torch.from_numpy(b))
    batch.solve()
    torch.cuda.synchronize()
    assert int(batch.info.abs().sum()) == 0
    return batch.A.cpu().numpy(), batch.B.cpu().numpy()


COUNT = 100_000


def test_quotients():
    rng = np.random.default_rng(1)
    a, b = numbers(rng, COUNT), numbers(rng, COUNT)
    rng.shuffle(b)
    a *= np.where(rng.random(COUNT) < 0.5, -1.0, 1.0)
    b[:50] = 0.0
    _, x = solve(np.ones(COUNT, np.int32), np.zeros(COUNT, np.int32), a, b)
    with np.errstate(all="ignore"):
        assert same(x, b / a)


def test_quotients_beside_a_midpoint():
    """b / a with b = a q rounded, q a 53-bit significand and a half: the exact quotient is next to a midpoint."""
    rng = np.random.default_rng(2)
    a = 1.0 + rng.integers(0, 2**52, COUNT) * 2.0**-52
    q = 1.0 + rng.integers(0, 2**52, COUNT) * 2.0**-52
    b = a * q + a * 2.0**-53  # within an ulp of a (q + half an ulp)
    b = np.nextafter(b, np.where(rng.random(COUNT) < 0.5, 0.0, 8.0))
    _, x = solve(np.ones(COUNT, np.int32), np.zeros(COUNT, np.int32), a, b)
    assert same(x, b / a)


def test_reciprocals():
    rng = np.random.default_rng(3)
    d = numbers(rng, COUNT)
    d = np.where(np.isinf(d), 1.5, d)
    s = np.ldexp(1.0, np.frexp(d)[1] - 1)  # a power of two, not above d: row 1 stays the pivot's
    a = np.zeros((COUNT, 4))
    a[:, 0], a[:, 1], a[:, 3] = d, s, 1.0  # column-major 2 x 2
    f, _ = solve(np.full(COUNT, 2, np.int32), np.zeros(COUNT, np.int32), a.reshape(-1), np.zeros(2 * COUNT))
    with np.errstate(all="ignore"):
        assert same(np.ascontiguousarray(f.reshape(COUNT, 4)[:, 1]), s * (1.0 / d))


def test_square_roots():
    rng = np.random.default_rng(4)
    d = numbers(rng, COUNT)
    # squares of 27-bit numbers and their neighbours: exact roots, and roots beside them
    r = rng.integers(2**26, 2**27, COUNT // 4).astype(np.float64)
    d[100:100 + r.size] = np.where(rng.random(r.size) < 0.5, r * r, np.nextafter(r * r, np.inf))
    b = numbers(rng, COUNT)
    f, x = solve(np.ones(COUNT, np.int32), np.ones(COUNT, np.int32), d, b)
    with np.errstate(all="ignore"):
        root = np.sqrt(d)
        assert same(f, root)
        assert same(x, b / root / root)
