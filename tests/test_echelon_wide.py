"""Echelon forms of few rows and many columns, on both sides of the lines between the two ways to U12
(one product, or substitution for wide panels), in one panel and in several.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("p", [37, 251, 65521, 65537, 2147483647])
@pytest.mark.parametrize("m,n", [(3, 20000), (16, 16065), (16, 16064), (17, 16100), (48, 6065), (49, 6065), (60, 12065),
                                 (64, 12064), (130, 6300)])
def test_wide(cuda, p, m, n):
    A = gen.dense_zp(m, m, n, p)
    if m > 20:
        A[m // 2:m // 2 + 3] = A[:3]  # dependent rows
    want, rank, det = oracle.echelon_zp(p, A)
    got, r, d = cuda.echelonize(p, A.copy())
    assert (r, d) == (rank, det)
    assert np.array_equal(got, want)
