"""The triangular solve at the edges of its leaf choice (64-row inverses, their merging into 512-row
ones, one-launch leaves), for both reductions of the CUDA-core kernels.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("p", [65521, 65537, 2147483647])
@pytest.mark.parametrize("m,n", [(64, 5), (65, 33), (127, 70), (128, 1), (129, 64), (255, 40), (257, 65),
                                 (449, 31), (513, 20), (577, 3)])
def test_leaf_edges(cuda, m, n, p):
    for upper in (False, True):
        for unit in (False, True):
            U = gen.upper_zp(m, m, p, unit=unit)
            A = U if upper else np.ascontiguousarray(U.T)
            B = gen.dense_zp(n, m, n, p)
            want, bad = oracle.trsm_zp(p, A, B, upper, unit, 3)
            assert bad is None
            for kernel in (0, 2):
                cuda.set_trsm_kernel(kernel)
                try:
                    got = cuda.trsm(p, 3, A, B.copy(), upper, unit)
                finally:
                    cuda.set_trsm_kernel(0)
                assert np.array_equal(got, want), (upper, unit, kernel)
