"""Launches whose CTAs get an SM each: no more clusters than the device holds at once, or they would run in two
turns where CTAs that share SMs run in one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib
P = C.POINTER(C.c_double)


def test_no_more_than_fit():
    """Clusters of one and two CTAs fill the chip; larger ones leave part of each group of SMs unused."""
    ctx = ttcuda.get_context()
    n, sms = C.c_int(), C.c_int()
    held = {}
    for csize in (1, 2, 4, 8):
        ctx.check(lib.ttc_test_lone_clusters(ctx.h, csize, C.byref(n), C.byref(sms)))
        held[csize] = n.value
        assert 1 <= n.value * csize <= sms.value
    assert held[1] == sms.value and held[8] <= held[4] // 2 <= held[2] // 4


@pytest.mark.parametrize("n,csize", [(256, 8), (128, 4)])
def test_clusters_of_all_sms_run_in_one_turn(n, csize):
    """From 80 % of the SMs up to all of them in clusters: where not every cluster fits with SMs of its own, CTAs
    share SMs.  (Two turns take twice the time of a few clusters, sharing 1.2 to 1.4 times; the bound lies
    between.)"""
    ctx = ttcuda.get_context()
    held, sms = C.c_int(), C.c_int()
    ctx.check(lib.ttc_test_lone_clusters(ctx.h, csize, C.byref(held), C.byref(sms)))
    g = np.random.default_rng(n)
    R = np.linalg.qr(g.standard_normal((n, n)) * 10.0 ** (-np.arange(n) / 32.0))[1].T.ravel(order="F")

    def ms(count):
        X, t, sweeps = np.tile(R, count), C.c_double(), np.zeros(count, np.int32)
        best = np.inf
        for _ in range(5):
            ctx.check(lib.ttc_test_jacobi_bench(ctx.h, C.c_int(count), C.c_int(n), C.c_int(n), X.ctypes.data_as(P), C.c_int(4),
                                                C.byref(t), sweeps.ctypes.data_as(C.POINTER(C.c_int))))
            best = min(best, t.value)
        return best

    few, full = ms(4), sms.value // csize
    for count in range(full * 4 // 5, full + 1):
        assert ms(count) <= 1.7 * few, count
