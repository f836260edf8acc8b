"""The dense Faugere-Lachartre output at row starts and widths off the 16-byte grid, and the columns
gathered for it at row counts around the eight a thread takes, and widths around the 4096 columns put together at once.  Exact against the CPU oracle; entries
around the output stay as they are."""
import types

import numpy as np
import pytest

import oracle
from lela_b200 import gen


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(7, 9), (8, 11), (17, 20), (41, 49), (331, 398), (60, 4095), (60, 4097), (90, 8190)])
@pytest.mark.parametrize("pad,off", [(1, 0), (2, 1), (4, 3), (7, 2)])
def test_fl_output_alignment(cuda, m, n, pad, off):
    import torch
    p = 65521
    X = gen.f4_matrix(m, m, p, n=n)
    T = types.SimpleNamespace(m=X.m, n=X.n, rowptr=torch.from_numpy(X.rowptr.view(np.int64)).cuda(),
                              colidx=torch.from_numpy(X.colidx.view(np.int32)).cuda(),
                              vals=torch.from_numpy(X.vals.view(np.int32)).cuda())
    for red, od in ((1, 0), (0, 0), (1, 1), (0, 1)):
        want = oracle.fl_echelonize_zp(p, X.m, X.n, X.rowptr, X.colidx, X.vals, red, od)
        full = torch.full((m, n + pad), -7, device="cuda", dtype=torch.int32)
        R = full[:, off:off + n]
        torch.cuda.synchronize()
        got, rank, det = cuda.fl_echelonize(p, T, bool(red), bool(od), R=R)
        torch.cuda.synchronize()
        assert (rank, det) == (want["rank"], want["det"])
        rows = want["R"].shape[0]
        assert np.array_equal(R.cpu().numpy().view(np.uint32)[:rows], want["R"])
        out = full.cpu().numpy()
        assert (out[:, :off] == -7).all() and (out[:, off + n:] == -7).all()
