"""Products whose C lies over A or B on the device: the operands are split before C is written, so the
product is that of the operands as they were.  Exact against the CPU oracle; with C beside them in one
matrix, too."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


def views(X, width, boxes):
    """Views of one device matrix (rows, columns, row offset, column offset), and their residues."""
    import torch
    t = torch.from_numpy(X.view(np.int32)).cuda()
    assert t.shape[1] == width
    torch.cuda.synchronize()
    return t, [t[r:r + m, c:c + n] for m, n, r, c in boxes], [X[r:r + m, c:c + n].copy() for m, n, r, c in boxes]


# (A, B, C) as boxes of one matrix: rows, columns, first row, first column
BOXES = {
    "C is A": ((600, 200, 0, 0), (200, 200, 600, 3), (600, 200, 0, 0)),
    "C is B": ((200, 200, 600, 3), (200, 600, 0, 0), (200, 600, 0, 0)),
    "C over part of A": ((600, 200, 0, 0), (200, 300, 600, 0), (600, 300, 130, 70)),
    "C over the ends of B's rows": ((200, 200, 600, 3), (200, 300, 0, 0), (200, 300, 1, 290)),
    "C beside both": ((200, 200, 0, 0), (200, 300, 200, 0), (200, 300, 0, 250)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("p", [251, 65521, 2147483647])
@pytest.mark.parametrize("boxes", list(BOXES.values()), ids=list(BOXES))
@pytest.mark.parametrize("a,b", [(1, 0), (3, 2)])
def test_overlap(cuda, p, boxes, a, b):
    X = gen.dense_zp(p % 100, 900, 640, p)
    t, (A, B, C), (hA, hB, hC) = views(X, 640, boxes)
    cuda.gemm(p, a, A, B, b, C)
    cuda.synchronize()
    want = X.copy()
    m, n, r, c = boxes[2]
    want[r:r + m, c:c + n] = oracle.gemm_zp(p, hA, hB, hC, a, b)
    assert np.array_equal(t.cpu().numpy().view(np.uint32), want)


@pytest.mark.gpu
def test_overlap_in_row_blocks(cuda):
    """A product by residues whose planes need several row blocks, C one row after A's first."""
    import torch
    p, m, k = 4294967291, 9500, 32768
    g = torch.Generator(device="cuda").manual_seed(6)
    rand = lambda *s: torch.randint(-2**31, 2**31 - 8, s, generator=g, device="cuda", dtype=torch.int32)  # noqa: E731
    X, B = rand(m + 128, k), rand(k, 4096)
    A, C = X[:m], X[128:, :4096]
    rows = [0, 1, 4863, 4864, 4991, 4992, 6000, m - 1]
    res = lambda t: t.cpu().numpy().view(np.uint32) % np.uint32(p)  # noqa: E731
    hA = res(A[rows])
    torch.cuda.synchronize()
    cuda.gemm(p, 1, A, B, 0, C)
    cuda.synchronize()
    assert np.array_equal(C[rows].cpu().numpy().view(np.uint32),
                          oracle.gemm_zp(p, hA, res(B), np.zeros((len(rows), 4096), np.uint32), 1, 0, threads=8))
