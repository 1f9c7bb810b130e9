"""Grouped FP64 GEMM with K split: adding up the partial tiles is a small part of the launch."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
P, L = C.POINTER(C.c_double), C.c_longlong


def ms(m, n, k, batch):
    ctx = ttcuda.get_context()
    g = np.random.default_rng(1)
    A, B, c = g.standard_normal(m * k * batch), g.standard_normal(k * n * batch), np.zeros(m * n * batch)
    strides = [(L * 5)(*v) for v in ((1, 0, m, 0, m * k), (1, 0, k, 0, k * n), (1, 0, m, 0, m * n))]
    best = np.inf
    for _ in range(6):
        ctx.set_profiling(True)
        ctx.check(ttcuda.lib.ttc_test_gemm(ctx.h, *map(C.c_int, (m, n, k, batch, m, n, k)), A.ctypes.data_as(P), L(A.size), strides[0],
                                           B.ctypes.data_as(P), L(B.size), strides[1], c.ctypes.data_as(P), L(c.size), strides[2],
                                           C.c_double(1.0), C.c_double(0.0)))
        best = min(best, ctx.kernel_profile()["gemm_f64"][0])
        ctx.set_profiling(False)
    return best


def test_split_costs_little():
    """512 x 256 x 4096 in eight splits against eight products of 512 x 256 x 512: the same tiles and products.
    The partials are 8 MB, written once and read once through L2, 2 us at 8 TB/s, by an eighth of the CTAs, after
    50 us of products: a quarter more covers the latency of reading them."""
    assert ms(512, 256, 4096, 1) <= 1.25 * ms(512, 256, 512, 8)
