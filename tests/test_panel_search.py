"""The echelon panel's pivot search at the edges of its three field arithmetics (signed residues for
32 <= p <= 65521, Montgomery products for the other odd p < 2^31, Barrett products else), on windows
that fill, overflow and run out.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen

PRIMES = [2, 3, 29, 31, 37, 251, 257, 16381, 16411, 32749, 32771, 65519, 65521, 65537, 2147483647]
# moduli with zero divisors or past 2^31: matrices whose pivots are all 1
UNIT_PIVOTS = [32, 63, 64, 65520, 65522, 65535, 65536, 2147483646, 2147483648, 4294967291]


def _check(cuda, p, A):
    want, wr, wd = oracle.echelon_zp(p, A)
    got, gr, gd = cuda.echelonize(p, A.copy())
    assert (gr, gd) == (wr, wd)
    assert np.array_equal(got, want)


def _staircase(g, A, p):
    """Rows sorted by leading column, as a Schur complement of the F4 step, some of them dependent."""
    m, n = A.shape
    head = np.sort(g.integers(0, n, size=m))
    A[np.arange(n)[None, :] < head[:, None]] = 0
    for r in g.choice(m, size=m // 12, replace=False):
        a = int(g.integers(0, m))
        A[r] = A[a].astype(np.uint64) * 3 % p
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("p", PRIMES)
def test_primes(cuda, p):
    g = np.random.default_rng(p)
    for m, n in ((79, 64), (81, 63), (17, 130), (900, 129)):
        _check(cuda, p, gen.dense_zp(m + n, m, n, p))
    _check(cuda, p, np.full((97, 66), p - 1, dtype=np.uint32))
    _check(cuda, p, _staircase(g, gen.dense_zp(5, 400, 300, p), p))
    A = gen.dense_zp(6, 300, 140, p)
    A[:150, :50] = 0  # pivots past a window that has rows without one
    A[150:, 3:20] = 0
    A[10:140:3, 40:60] = 0
    _check(cuda, p, A)


@pytest.mark.gpu
@pytest.mark.parametrize("p", UNIT_PIVOTS)
def test_other_moduli(cuda, p):
    g = np.random.default_rng(p)
    for m, n in ((64, 64), (130, 100)):
        L = np.tril(g.integers(0, p, size=(m, n), dtype=np.uint64), -1)
        U = np.triu(g.integers(0, p, size=(n, n), dtype=np.uint64), 1)
        L[np.arange(n), np.arange(n)] = 1
        U[np.arange(n), np.arange(n)] = 1
        A = np.array([[int(sum(int(a) * int(b) for a, b in zip(L[i], U[:, j]))) % p for j in range(n)]
                      for i in range(m)], dtype=np.uint32)
        _check(cuda, p, A)
