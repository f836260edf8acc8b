"""An echelon form after a call that failed.  The form waits on the host between panels, so it cannot
be captured: a call on a capturing stream fails, and its kernels have not run.  What the handle keeps
must be what has run: the next form modulo the same p is exact against the CPU oracle."""
import ctypes

import numpy as np
import pytest

import oracle
from lela_b200 import CudaModule, gen
from lela_b200.api import CudaError

RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED


@pytest.mark.gpu
@pytest.mark.parametrize("before,p", [(65521, 101), (251, 32771)])
def test_form_after_captured_call(before, p):
    import torch
    driver = ctypes.CDLL("libcuda.so.1")
    m, n = 90, 110
    A = gen.dense_zp(1, m, n, p)
    want, rank, det = oracle.echelon_zp(p, A)
    stream = torch.cuda.Stream()
    handle = ctypes.c_void_p(stream.cuda_stream)
    with CudaModule(0) as cm:
        cm.set_stream(stream)
        # the handle's buffers exist before the capture
        cm.echelonize(before, torch.from_numpy(gen.dense_zp(2, m, n, before).view(np.int32)).cuda())
        dA = torch.from_numpy(A.view(np.int32)).cuda()
        torch.cuda.synchronize()
        assert driver.cuStreamBeginCapture_v2(handle, RELAXED) == 0
        try:
            with pytest.raises(CudaError):
                cm.echelonize(p, dA)
        finally:
            graph = ctypes.c_void_p()
            driver.cuStreamEndCapture(handle, ctypes.byref(graph))
            if graph.value:
                driver.cuGraphDestroy(graph)
        torch.cuda.synchronize()
        for _ in range(2):
            dA = torch.from_numpy(A.view(np.int32)).cuda()
            torch.cuda.synchronize()
            _, r, d = cm.echelonize(p, dA)
            cm.synchronize()
            assert (r, d) == (rank, det)
            assert np.array_equal(dA.cpu().numpy().view(np.uint32), want)
