"""The reciprocal and the reciprocal square root of the factorisations' kernels against 64-bit mantissas, over
the ranges that they are stated for."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
P = C.POINTER(C.c_double)
U = 2.0 ** -53


def device(x):
    x = np.ascontiguousarray(x)
    rs, rc = np.empty_like(x), np.empty_like(x)
    ctx = ttcuda.get_context()
    ctx.check(ttcuda.lib.ttc_test_reciprocals(ctx.h, x.size, *(a.ctypes.data_as(P) for a in (x, rs, rc))))
    return rs, rc


def values(lo, hi):
    """Mantissas of every kind (random, at both ends of a binade, beside 1 and 2) at every exponent in [lo, hi)."""
    g = np.random.default_rng(lo & 0xffff)
    e = np.arange(lo, hi)
    m = [g.uniform(1.0, 2.0, e.size) for _ in range(200)]
    m += [np.full(e.size, v) for v in (1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5, np.sqrt(2.0))]
    return np.concatenate([np.ldexp(v, e) for v in m])


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs the 80-bit format")
def test_against_long_double():
    x = values(-1022, 1000)
    want = 1 / np.sqrt(x.astype(np.longdouble))
    assert (np.abs(device(x)[0] - want) <= 1.7 * U * want).all()
    x = values(-1000, 1000)
    x[1::2] *= -1.0
    want = 1 / x.astype(np.longdouble)
    assert (np.abs(device(x)[1] - want) <= 1.1 * U * np.abs(want)).all()
