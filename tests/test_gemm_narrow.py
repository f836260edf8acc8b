"""Products of few terms over many rows or columns: the split's shared warps (rows of at most 64
columns), and the kernel that wide products of few rows go to.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("p", [251, 65521, 2147483647])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65])
@pytest.mark.parametrize("m", [1003, 16383, 16389])
def test_short_rows(cuda, p, k, m):
    n = 70
    A, B, C = gen.dense_zp(1, m, k, p), gen.dense_zp(2, k, n, p), gen.dense_zp(3, m, n, p)
    cuda.set_gemm_kernel(2)
    try:
        got = cuda.gemm(p, p - 1, A, B, 1, C.copy())
    finally:
        cuda.set_gemm_kernel(0)
    assert np.array_equal(got, oracle.gemm_zp(p, A, B, C, p - 1, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("p", [251, 65521, 2147483647])
@pytest.mark.parametrize("m,n,k", [(1, 50001, 5), (33, 40003, 32), (64, 40003, 16), (64, 40003, 17), (64, 30000, 32),
                                   (65, 30000, 5), (20, 40000, 33), (30000, 5, 7)])
def test_wide(cuda, p, m, n, k):
    A, B, C = gen.dense_zp(4, m, k, p), gen.dense_zp(5, k, n, p), gen.dense_zp(6, m, n, p)
    got = cuda.gemm(p, 3, A, B, 2, C.copy())
    assert np.array_equal(got, oracle.gemm_zp(p, A, B, C, 3, 2, threads=8))
