"""ttc_qr_noalloc under a caller's stream capture: the nodes that it adds to the caller's graph hang together
by plain dependencies, which every query of a graph can return."""
import ctypes as C

import numpy as np
import pytest

import torch

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib


def test_edges_are_plain():
    driver = C.CDLL("libcuda.so.1")
    m, n = 40, 12
    A = torch.randn(n, m, dtype=torch.float64, device="cuda")
    Q, R = torch.zeros(m * n, dtype=torch.float64, device="cuda"), torch.zeros(n * n, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    args = (m, n, A.data_ptr(), m, Q.data_ptr(), m, R.data_ptr(), n, status.data_ptr())
    lib.ttc_qr_noalloc.argtypes = [C.c_int32, C.c_int32, C.c_void_p, C.c_int64, C.c_void_p, C.c_int64, C.c_void_p, C.c_int64,
                                   C.c_void_p, C.c_void_p]
    assert lib.ttc_qr_noalloc(*args, stream.cuda_stream) == 0       # resolves the scratch array's address
    torch.cuda.synchronize()
    want = Q.clone(), R.clone()
    s, graph, count = C.c_void_p(stream.cuda_stream), C.c_void_p(), C.c_size_t(0)
    assert driver.cuStreamBeginCapture_v2(s, 1) == 0
    rc = lib.ttc_qr_noalloc(*args, stream.cuda_stream)
    assert driver.cuStreamEndCapture(s, C.byref(graph)) == 0 and rc == 0
    try:
        assert driver.cuGraphGetEdges(graph, None, None, C.byref(count)) == 0 and count.value >= 2
        a, b = (C.c_void_p * count.value)(), (C.c_void_p * count.value)()
        assert driver.cuGraphGetEdges(graph, a, b, C.byref(count)) == 0
        ex = C.c_void_p()
        assert driver.cuGraphInstantiateWithFlags(C.byref(ex), graph, C.c_ulonglong(0)) == 0
        Q.zero_()
        R.zero_()
        torch.cuda.synchronize()
        assert driver.cuGraphLaunch(ex, s) == 0
        torch.cuda.synchronize()
        assert torch.equal(Q, want[0]) and torch.equal(R, want[1]) and int(status) == 0
        driver.cuGraphExecDestroy(ex)
    finally:
        driver.cuGraphDestroy(graph)
