"""The smallest Z/p products, on both sides of the line between the CUDA-core kernel for small K and
the one-launch tensor-core kernel.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 251, 257, 65521, 65537])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 16, 32), (16, 17, 32), (17, 16, 32), (16, 16, 33), (32, 32, 32),
                                   (33, 32, 32), (16, 64, 31), (1000, 16, 32), (1025, 16, 32), (5, 3000, 7)])
def test_smallest(cuda, p, m, n, k):
    import torch
    A, B, C = gen.dense_zp(1, m, k, p), gen.dense_zp(2, k, n, p), gen.dense_zp(3, m, n, p)
    for a, b in ((1, 0), (p - 1, 1), (3 % p, 2 % p)):
        full = torch.full((m, n + 3), -7, dtype=torch.int32, device="cuda")
        dC = full[:, 1:1 + n]
        dC.copy_(torch.from_numpy(C.view(np.int32)))
        dA, dB = (torch.from_numpy(x.view(np.int32)).cuda() for x in (A, B))
        torch.cuda.synchronize()
        for _ in range(2):  # one behind the other on the stream
            cuda.gemm(p, a, dA, dB, b, dC)
        cuda.synchronize()
        want = oracle.gemm_zp(p, A, B, oracle.gemm_zp(p, A, B, C, a, b), a, b)
        assert np.array_equal(dC.cpu().numpy().view(np.uint32), want)
        out = full.cpu().numpy()
        assert (out[:, 0] == -7).all() and (out[:, 1 + n:] == -7).all()
