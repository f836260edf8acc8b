"""Device-pointer calls captured into a CUDA graph, whose kernels are launched early one behind the other:
replayed on new inputs they give what the calls give.  A call whose larger planes the workspace cannot hold
without growing takes the smaller ones there.  Exact against the CPU oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import CudaModule, gen

P16, P31 = 65521, 2147483647


def put(t, X):
    import torch
    t.copy_(torch.from_numpy(X.view(np.int64 if X.dtype == np.uint64 else np.int32)))


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k", [(251, 300, 300, 1100), (P16, 16, 16, 32), (P16, 64, 900, 64), (P16, 520, 513, 700),
                                     (P31, 1537, 1539, 700), (P31, 200, 300, 64)])
@pytest.mark.parametrize("warm", ["the same call", "a smaller workspace"])
def test_gemm(p, m, n, k, warm):
    import torch
    A, B, C = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((m, k), (k, n), (m, n)))
    D = torch.zeros_like(C)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with CudaModule(0) as cm:
        cm.set_stream(stream)
        if warm == "the same call":
            cm.gemm(p, 3, A, B, 1, C)
        else:  # 17 MB: room for the limbs of all these shapes, not for the largest's residues
            X = torch.zeros((2048, 2048), dtype=torch.int32, device="cuda")
            cm.gemm(P16, 1, X, X.clone(), 0, X.clone())
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            cm.gemm(p, 3, A, B, 1, C)  # two in a row, the second on the first's result
            cm.gemm(p, p - 1, A, B, 2, C)
            D.copy_(C)
        for seed in (1, 2):
            hA, hB, hC = gen.dense_zp(seed, m, k, p), gen.dense_zp(seed + 5, k, n, p), gen.dense_zp(seed + 9, m, n, p)
            put(A, hA), put(B, hB), put(C, hC)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            want = oracle.gemm_zp(p, hA, hB, oracle.gemm_zp(p, hA, hB, hC, 3, 1), p - 1, 2)
            assert np.array_equal(D.cpu().numpy().view(np.uint32), want)
        del graph


@pytest.mark.gpu
def test_gemm_gf2():
    import torch
    m, n, k = 700, 900, 650
    A, B, C = (torch.zeros((r, (w + 63) // 64), dtype=torch.int64, device="cuda") for r, w in ((m, k), (k, n), (m, n)))
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with CudaModule(0) as cm:
        cm.set_stream(stream)
        cm.gemm_gf2(A, B, C, n, k)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            cm.gemm_gf2(A, B, C, n, k)
        for seed in (1, 2):
            hA, hB, hC = gen.dense_gf2(seed, m, k), gen.dense_gf2(seed + 5, k, n), gen.dense_gf2(seed + 9, m, n)
            put(A, hA), put(B, hB), put(C, hC)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(C.cpu().numpy().view(np.uint64), oracle.gemm_gf2(hA, hB, hC, k, n))
        del graph


@pytest.mark.gpu
def test_wide_solve_in_the_workspace_there_is():
    """A unit solve needs no host copy, so it can be captured; after a narrow solve the workspace (22 MB) holds the
    recursion's planes for the wide one (16 MB), not those of all of A and X (25 MB)."""
    import torch
    m, n = 2048, 3073
    A = torch.tril(torch.ones((4096, 4096), dtype=torch.int32, device="cuda"))
    B = torch.zeros((m, n), dtype=torch.int32, device="cuda")
    narrow = torch.zeros((4096, 200), dtype=torch.int32, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with CudaModule(0) as cm:
        cm.set_stream(stream)
        cm.trsm(P16, 1, A, narrow, False, True)
        T = A[:m, :m]
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            cm.trsm(P16, 1, T, B, False, True)
        hB = gen.dense_zp(3, m, n, P16)
        put(B, hB)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        # the inverse of the triangle of ones is the difference of neighbouring rows
        want = hB.astype(np.int64)
        want[1:] -= hB[:-1]
        assert np.array_equal(B.cpu().numpy().view(np.uint32), (want % P16).astype(np.uint32))
        del graph
