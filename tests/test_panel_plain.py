"""The echelon panel's pivot search in canonical residues (p = 2, other even moduli below 32 and above
65521), with 32-bit and with 64-bit reductions, on matrices of low rank, whose columns without a pivot
send it past its window.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 4, 30, 65522, 65534, 65536, 65538, 2147483648])
@pytest.mark.parametrize("m,n,r", [(200, 60, 54), (500, 130, 20), (300, 300, 100)])
def test_low_rank(cuda, p, m, n, r):
    # unit lower times unit upper: every pivot is 1, so that it can be inverted for any p
    g = np.random.default_rng(p + m)
    L = np.tril(g.integers(0, p, size=(m, r), dtype=np.uint64), -1)
    U = np.triu(g.integers(0, p, size=(r, n), dtype=np.uint64), 1)
    L[np.arange(r), np.arange(r)] = 1
    U[np.arange(r), np.arange(r)] = 1
    A = np.zeros((m, n), dtype=np.uint64)
    for k in range(r):
        A = (A + L[:, k:k + 1] * U[k:k + 1]) % np.uint64(p)
    cols = np.repeat(np.arange(n), 2)[:n]  # each column twice: every other one has no pivot
    A = np.ascontiguousarray(A[:, cols]).astype(np.uint32)
    want, wr, wd = oracle.echelon_zp(p, A)
    got, gr, gd = cuda.echelonize(p, A.copy())
    assert (gr, gd) == (wr, wd)
    assert np.array_equal(got, want)
