"""Products modulo p > 2^16 by residues: few moduli and the most, ragged tiles and K, the largest
entries, every way the result joins C, entries that are not reduced, and doubles.  Exact against the
CPU oracle, for shapes the automatic choice sends there and one on the other side of its line."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen

SHAPES = [
    # p, m, n, k
    (65537, 1153, 1031, 2049),
    (1000003, 2050, 1027, 2063),
    (2147483647, 1537, 1539, 1000),
    (4294967291, 1600, 1541, 905),
    (4294967291, 1536, 1536, 4096),
    (4294967291, 1535, 1700, 1000),
]


def on_device(x):
    import torch
    t = torch.zeros((x.shape[0], x.shape[1] + 3), device="cuda", dtype=torch.int32)
    t[:, 1:1 + x.shape[1]] = torch.from_numpy(x.view(np.int32))
    torch.cuda.synchronize()
    return t[:, 1:1 + x.shape[1]]


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k", SHAPES)
@pytest.mark.parametrize("largest", [False, True])
def test_gemm_residues(cuda, p, m, n, k, largest):
    A, B, C = gen.dense_zp(1, m, k, p), gen.dense_zp(2, k, n, p), gen.dense_zp(3, m, n, p)
    if largest:
        A[:] = p - 1
        B[:, 1::3] = p - 1
    R = oracle.gemm_zp(p, A, B, np.zeros_like(C), 1, 0, threads=8).astype(object)
    dA, dB = on_device(A), on_device(B)
    for a, b in ((1, 0), (5, 0), (1, 1), (p - 1, 1), (3, p - 2)):
        dC = on_device(C)
        cuda.gemm(p, a, dA, dB, b, dC)
        cuda.synchronize()
        assert np.array_equal(dC.cpu().numpy().view(np.uint32).astype(object), (R * a + C.astype(object) * b) % p)
    # the same entries, not reduced
    lift = A < 2**32 - p
    if lift.any():
        A[lift] += np.uint32(p)
        dC = on_device(C)
        cuda.gemm(p, 1, on_device(A), dB, 0, dC)
        cuda.synchronize()
        assert np.array_equal(dC.cpu().numpy().view(np.uint32).astype(object), R)


@pytest.mark.gpu
def test_gemm_residues_double(cuda):
    import torch
    p, m, n, k = 67108859, 1153, 1031, 2049
    X = [gen.dense_zp(s, *shape, p) for s, shape in ((1, (m, k)), (2, (k, n)), (3, (m, n)))]
    A, B, C = (oracle.from_residues(x, p, np.float64) for x in X)
    want = oracle.gemm_zp_elem(p, A, B, C, 1, p - 1)
    dC = torch.from_numpy(C).cuda()
    cuda.gemm(p, 1, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), p - 1, dC)
    cuda.synchronize()
    assert np.array_equal(dC.cpu().numpy(), want)


@pytest.mark.gpu
def test_gemm_residues_row_blocks(cuda):
    """Planes beyond one block's room (two row blocks): rows of each, around the line."""
    import torch
    p, m, n, k = 4294967291, 9500, 2048, 32768
    g = torch.Generator(device="cuda").manual_seed(5)
    A, B, C = (torch.randint(-2**31, 2**31 - 8, s, generator=g, device="cuda", dtype=torch.int32)
               for s in ((m, k), (k, n), (m, n)))
    C0 = C.clone()
    torch.cuda.synchronize()
    cuda.gemm(p, 3, A, B, 2, C)
    cuda.synchronize()
    rows = [0, 4735, 4736, 4751, 4863, 4864, 4991, 4992, m - 1]
    res = lambda t: t.cpu().numpy().view(np.uint32) % np.uint32(p)
    want = oracle.gemm_zp(p, res(A[rows]), res(B), res(C0[rows]), 3, 2, threads=8)
    assert np.array_equal(C[rows].cpu().numpy().view(np.uint32), want)
