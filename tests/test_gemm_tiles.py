"""The automatic tile choice of the Z/p gemm on both sides of its lines, the typed gemm on the tensor
cores (operands split from their own element type, C combined in one pass), and the GF(2) expansions
at ragged sizes.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,p", [
    (130, 300, 1030, 251),      # one limb, few tiles
    (2050, 1793, 1024, 251),    # one limb, wide tiles (17 x 8 of 148 SMs)
    (2050, 1793, 1023, 251),
    (520, 513, 512, 65521),     # two limbs, few tiles
    (1153, 1153, 512, 65521),   # 10 x 10 wide tiles
    (1153, 1153, 511, 65521),
])
def test_tile_choice(cuda, m, n, k, p):
    A, B, C = gen.dense_zp(1, m, k, p), gen.dense_zp(2, k, n, p), gen.dense_zp(3, m, n, p)
    want = oracle.gemm_zp(p, A, B, C, p - 1, 1, threads=8)
    cuda.set_gemm_kernel(2)
    try:
        got = cuda.gemm(p, p - 1, A, B, 1, C.copy())
    finally:
        cuda.set_gemm_kernel(0)
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,p", [(np.uint8, 251), (np.uint8, 2), (np.uint16, 251), (np.uint16, 65521),
                                     (np.float32, 4093), (np.float64, 67108859), (np.float64, 101)])
@pytest.mark.parametrize("a,b", [(1, 1), (3, 0), (1, 2)])
def test_typed_gemm(cuda, dtype, p, a, b):
    import torch
    a, b = a % p, b % p
    m, n, k = 333, 277, 515
    R = [gen.dense_zp(s, *shape, p) for s, shape in ((1, (m, k)), (2, (k, n)), (3, (m, n)))]
    A, B, C = (oracle.from_residues(x, p, dtype) for x in R)
    want = oracle.gemm_zp_elem(p, A, B, C, a, b)
    # odd strides and offsets on the device
    def view(x, pad):
        t = torch.zeros((x.shape[0], x.shape[1] + pad), device="cuda",
                        dtype=torch.from_numpy(x[:1].copy()).dtype)
        v = t[:, pad - 1:pad - 1 + x.shape[1]]
        v.copy_(torch.from_numpy(x))
        return t, v
    (_, vA), (_, vB), (tC, vC) = view(A, 3), view(B, 2), view(C, 5)
    torch.cuda.synchronize()
    cuda.set_gemm_kernel(2)
    try:
        cuda.gemm(p, a, vA, vB, b, vC)
        cuda.synchronize()
    finally:
        cuda.set_gemm_kernel(0)
    assert np.array_equal(vC.cpu().numpy(), want)
    assert not tC[:, :4].cpu().numpy().any() and not tC[:, 4 + n:].cpu().numpy().any()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (5, 64, 63), (70, 65, 129), (130, 321, 255), (9, 500, 1000)])
def test_gf2_expansion(cuda, m, n, k):
    A, B, C = gen.dense_gf2(1, m, k), gen.dense_gf2(2, k, n), gen.dense_gf2(3, m, n)
    want = oracle.gemm_gf2(A, B, C, k, n)
    cuda.set_gf2_kernel(1)
    try:
        got = cuda.gemm_gf2(A, B, C.copy(), n, k)
    finally:
        cuda.set_gf2_kernel(0)
    assert np.array_equal(got, want)
