"""Entries that are not reduced modulo p: a panel's entries are before its pivot search, which looks
inverses up by value (32 <= p <= 65521).  A form of one panel is that of the reduced matrix; one of
several ends, whatever its other kernels make of such entries, and the next form is right."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("p", [37, 251, 16381, 32771, 65521])
@pytest.mark.parametrize("top", [1 << 16, 1 << 20, 1 << 32])
@pytest.mark.parametrize("m,n", [(40, 64), (90, 50), (700, 33)])
def test_one_panel(cuda, p, top, m, n):
    g = np.random.default_rng(p + m)
    A = g.integers(0, top, size=(m, n), dtype=np.uint64)
    A[m // 3: m // 2] = A[0] * 3 % p     # dependent rows
    A[:m // 4, :5] = p                   # nonzero words of residue zero
    want, rank, det = oracle.echelon_zp(p, (A % p).astype(np.uint32))
    got, r, d = cuda.echelonize(p, A.astype(np.uint32))
    assert (r, d) == (rank, det)
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("p", [251, 65521])
def test_several_panels_end(cuda, p):
    A = np.random.default_rng(p).integers(0, 1 << 32, size=(700, 300), dtype=np.uint64).astype(np.uint32)
    _, r, _ = cuda.echelonize(p, A)
    assert 0 < r <= 300
    B = gen.dense_zp(5, 300, 200, p)
    want, rank, det = oracle.echelon_zp(p, B)
    got, r, d = cuda.echelonize(p, B.copy())
    assert (r, d) == (rank, det) and np.array_equal(got, want)
