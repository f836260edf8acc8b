"""Calls on a device with little free memory: what a handle keeps from one call must not stand in the
way of the next one's buffers.  The rest of the memory is taken by an allocation of the test's own, as by
another allocator of the program.  Results equal those with room, which other tests check."""
import numpy as np
import pytest

from lela_b200 import CudaModule, gen

MB = 1 << 20
P16, P31 = 65521, 2147483647


def rand(seed, m, n, p):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, p, (m, n), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def leave(room):
    """An allocation that leaves about `room` bytes of the device free."""
    import torch
    torch.cuda.empty_cache()
    filler = torch.empty(free() - room, dtype=torch.uint8, device="cuda")
    assert room - 8 * MB < free() < room + 8 * MB
    return filler


@pytest.fixture
def tidy():
    import torch
    yield
    torch.cuda.empty_cache()


@pytest.mark.gpu
def test_workspace_makes_room(tidy):
    """The planes of a product by residues (503 MB where limbs take 134) are in the workspace; the
    host-pointer product after it needs 432 MB of staging and 145 of planes."""
    import torch
    A, B = rand(1, 4096, 4096, P31), rand(2, 4096, 4096, P31)
    hA, hB, hC = (gen.dense_zp(s, 6000, 6000, P16) for s in (3, 4, 5))
    with CudaModule(0) as cm:
        C = A.clone()
        want = cm.gemm(P16, 1, hA, hB, 1, hC.copy())
        cm.gemm(P31, 1, A, B, 0, C)
        cm.synchronize()
        wantC = C.clone()
    with CudaModule(0) as cm:
        cm.gemm(P31, 1, A, B, 0, C)
        cm.synchronize()
        filler = leave(300 * MB)
        got = cm.gemm(P16, 1, hA, hB, 1, hC.copy())
        assert np.array_equal(got, want)
        C.zero_()
        cm.gemm(P31, 1, A, B, 0, C)  # with what is left
        cm.synchronize()
        del filler
    torch.cuda.empty_cache()
    assert bool((C == wantC).all())


@pytest.mark.gpu
def test_fl_after_its_wide_solve(tidy):
    """Faugere-Lachartre at a size whose solve keeps the planes of all of A and X (86 MB where the
    recursion and the Schur complement take 54), and the reduced form's blocks (108 MB) come after: 16 MB
    less than the call would hold if both stayed."""
    import torch
    import types
    X = gen.f4_matrix_fast(1, 6000, P16, n=9000, density=0.01)
    D = types.SimpleNamespace(m=X.m, n=X.n, rowptr=torch.from_numpy(X.rowptr.view(np.int64)).cuda(),
                              colidx=torch.from_numpy(X.colidx.view(np.int32)).cuda(),
                              vals=torch.from_numpy(X.vals.view(np.int32)).cuda())
    R, want = (torch.zeros((X.m, X.n), dtype=torch.int32, device="cuda") for _ in range(2))
    for _ in range(2):  # the first call loads the kernels, the second shows what a call holds
        with CudaModule(0) as cm:
            torch.cuda.empty_cache()
            before = free()
            _, rank, det = cm.fl_echelonize(P16, D, R=want)
            cm.synchronize()
            held = before - free()
    with CudaModule(0) as cm:
        filler = leave(held - 16 * MB)
        _, r, d = cm.fl_echelonize(P16, D, R=R)
        cm.synchronize()
        del filler
    torch.cuda.empty_cache()
    assert (r, d) == (rank, det)
    assert bool((R == want).all())


@pytest.mark.gpu
def test_planes_leave_memory_free(tidy):
    """With less than a sixteenth of the device free, a product modulo p > 2^16 and a wide solve take
    the workspace of the limbs (134 MB, where the residue planes have 503) and of the recursion (42 MB and
    the inverses, where the planes of all of A and X have 67 and their leaf's)."""
    import torch
    A, B = rand(1, 4096, 4096, P31), rand(2, 4096, 4096, P31)
    T = torch.tril(rand(3, 4096, 4096, P16), -1) + torch.eye(4096, device="cuda", dtype=torch.int32)
    Y = rand(4, 4096, 4096, P16)

    def run(op):
        C = Y.clone()
        torch.cuda.synchronize()
        before = free()
        with CudaModule(0) as cm:
            if op == "gemm":
                cm.gemm(P31, 1, A, B, 0, C)
            else:
                cm.trsm(P16, 1, T, C, False, True)
            cm.synchronize()
            return before - free(), C

    run("gemm"), run("trsm")  # the kernels
    roomy = {op: run(op) for op in ("gemm", "trsm")}
    filler = leave(6 << 30)
    tight = {op: run(op) for op in ("gemm", "trsm")}
    del filler
    assert tight["gemm"][0] < 144 * MB < roomy["gemm"][0]
    assert tight["trsm"][0] < roomy["trsm"][0] - 16 * MB
    for op in tight:
        assert bool((tight[op][1] == roomy[op][1]).all())


@pytest.mark.gpu
def test_fl_batch_keeps_its_budget(tidy):
    """Two wide matrices modulo 2^31 - 1 at once, in a budget of twice the estimate that the header gives:
    their last product's residue planes (845 MB) are not in it and must not be taken."""
    import torch
    import types
    m, n = 5000, 20000
    Xs, outs = [], []
    for i in range(2):
        X = gen.f4_matrix_fast(i, m, P31, n=n, density=0.002)
        Xs.append(types.SimpleNamespace(m=m, n=n, rowptr=torch.from_numpy(X.rowptr.view(np.int64)).cuda(),
                                        colidx=torch.from_numpy(X.colidx.view(np.int32)).cuda(),
                                        vals=torch.from_numpy(X.vals.view(np.int32)).cuda()))
    budget = 2 * (4 * m * n + 4 * (m + n) * m + 5120 * m + 256 * MB)
    for limit in (0, budget):  # (the first call loads the kernels, too)
        Rs = [torch.zeros((m, n), dtype=torch.int32, device="cuda") for _ in Xs]
        torch.cuda.empty_cache()
        before = free()
        with CudaModule(0) as cm:
            cm.set_batch_memory_budget(limit)
            res = cm.fl_echelonize_batch(Xs, [P31, P31], Rs, True, nworkers=2)
            cm.synchronize()
            held = before - free()
        outs.append((Rs, res))
    assert outs[0][1] == outs[1][1]
    assert all(bool((a == b).all()) for a, b in zip(outs[0][0], outs[1][0]))
    assert held <= budget
