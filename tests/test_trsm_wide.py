"""The triangular solve leaf by leaf (wide right-hand sides): a last leaf of one row, of as many as the
one-launch kernel takes and of more, upper and lower, unit and not, with a factor, at odd strides, with
one, two and four limbs, and for a sparse A with leaves that nothing before them touches.  A X = a B,
exactly, in float64 products of at most 2^44; X reduced."""
import numpy as np
import pytest



def rand(seed, m, n, p):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, p, (m, n), generator=g, device="cuda", dtype=torch.int64)


def product(A, X, p):
    """A X mod p of int64 residues."""
    import torch
    if p <= 1 << 16:
        return (A.double() @ X.double()).to(torch.int64) % p
    a1, a0, x1, x0 = ((t >> s & 65535).double() for t in (A, X) for s in (16, 0))
    parts = [(u @ v).to(torch.int64) % p for u, v in ((a1, x1), (a1, x0), (a0, x1), (a0, x0))]
    return ((parts[0] * 65536 % p + parts[1] + parts[2]) % p * 65536 + parts[3]) % p


def strided(X, pad):
    """X as a view with row stride columns + pad and an odd start."""
    import torch
    full = torch.full((X.shape[0], X.shape[1] + pad), -7, dtype=torch.int32, device="cuda")
    full[:, 1:1 + X.shape[1]] = X.to(torch.int32)
    return full, full[:, 1:1 + X.shape[1]]


def check(A, X, B, a, p):
    assert int(X.min()) >= 0 and int(X.max()) < p
    assert bool((product(A, X, p) == B * a % p).all())


@pytest.mark.gpu
@pytest.mark.parametrize("p", [251, 65521])
@pytest.mark.parametrize("m", [2048, 2049, 2176, 2400])
@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("unit", [False, True])
def test_wide(cuda, p, m, upper, unit):
    import torch
    n, a = 3073, 3
    A = rand(m, m, m, p)
    A = torch.triu(A, 1) if upper else torch.tril(A, -1)
    A += torch.diag(torch.ones(m, dtype=torch.int64, device="cuda") if unit else 1 + rand(5, 1, m, p - 1)[0])
    B = rand(m + 1, m, n, p)
    (_, vA), (full, vB) = strided(A, 3), strided(B, 2)
    torch.cuda.synchronize()
    cuda.trsm(p, a, vA, vB, upper, unit)
    cuda.synchronize()
    check(A, vB.to(torch.int64), B, a, p)
    assert bool((full[:, 0] == -7).all()) and bool((full[:, -1] == -7).all())


@pytest.mark.gpu
@pytest.mark.parametrize("p,n,cols", [(65521, 2561, 3073), (2147483647, 4097, 770), (2147483647, 4224, 800)])
def test_wide_sparse(cuda, p, n, cols):
    import torch
    g = np.random.default_rng(n)
    rp, ci, va = [0], [], []
    for r in range(n):
        # rows of the second and fourth leaf stay inside their leaf, the others reach some way on
        end = (r // 512 + 1) * 512 if r // 512 in (1, 3) else r + 900
        c = r + 1 + np.flatnonzero(g.random(max(0, min(n, end) - r - 1)) < 0.02)
        ci.append(np.concatenate([[r], c]))
        va.append(g.integers(1, p, len(c) + 1))
        rp.append(rp[-1] + len(c) + 1)
    rp, ci, va = np.array(rp), np.concatenate(ci), np.concatenate(va)
    A = torch.zeros((n, n), dtype=torch.int64, device="cuda")
    A[torch.from_numpy(np.repeat(np.arange(n), np.diff(rp))).cuda(), torch.from_numpy(ci).cuda()] = torch.from_numpy(va).cuda()
    B = rand(n, n, cols, p)
    X = B.to(torch.int32)
    torch.cuda.synchronize()
    cuda.trsm_csr_upper(p, 5, n, torch.from_numpy(rp).cuda(), torch.from_numpy(ci.astype(np.int32)).cuda(),
                        torch.from_numpy(va.astype(np.uint32).view(np.int32)).cuda(), X)
    cuda.synchronize()
    check(A, X.to(torch.int64) & 0xffffffff, B, 5, p)
