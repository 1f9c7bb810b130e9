"""Conversions to BF16 and TF32 at the edges of the transposing tiles, and element-wise launches of more
problems than the chip has blocks (one block per problem, striding over it)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib
L = C.c_longlong
lib.ttc_test_cvt.argtypes = [C.c_void_p, C.c_int, C.c_int, L, L, L, L, C.c_int, C.c_int, C.POINTER(C.c_double), L, C.c_void_p, L]


@pytest.mark.parametrize("rows,cols", [(1, 1), (15, 40), (16, 16), (31, 33), (32, 32), (33, 64), (100, 17), (257, 130)])
@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("count", [1, 3000])
def test_conversion(rows, cols, tf32, trans, count):
    """Integers below 256 are the same in every format; what lies between the rows stays as it was."""
    if count > 1 and rows * cols > 2000:
        pytest.skip("one small size is enough")
    g = np.random.default_rng(rows * cols)
    ld, ldd = rows + 3, (cols if trans else rows) + 5
    src = g.integers(-255, 256, (cols, ld)).astype(float)
    size = (rows if trans else cols) * ldd
    dst = np.full((count, size), 77, np.float32 if tf32 else np.uint16)
    ds = (ldd, 1) if trans else (1, ldd)
    ctx = ttcuda.get_context()
    ctx.check(lib.ttc_test_cvt(ctx.h, rows, cols, 1, ld, ds[0], ds[1], count, tf32, src.ctypes.data_as(C.POINTER(C.c_double)),
                               src.size, dst.ctypes.data, size * dst.itemsize))
    want = np.full(((rows if trans else cols), ldd), 77, dst.dtype)
    vals = src[:, :rows].T if trans else src[:, :rows]
    want[:, :vals.shape[1]] = vals if tf32 else (vals.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    assert (dst.reshape(count, *want.shape) == want).all()


def test_more_trains_than_blocks():
    """2500 trains rounded together at tolerance 0: each one is again the tensor that it was."""
    g = np.random.default_rng(1)
    dims, count = (3, 2, 4), 2500
    r = [1, 3, 2, 1]
    cores = [g.standard_normal((count, dims[k], r[k], r[k + 1])) for k in range(3)]
    vec = [ttcuda.TTvector(3, [np.asfortranarray(c[t]) for c in cores], dims, r) for t in range(count)]
    xb = ttcuda.DeviceBatch.from_tts(vec)
    yb = ttcuda.DeviceBatch(dims, [r] * count)
    xb.round_det(yb, tol=0.0)
    out = yb.download()

    def full(a, b, c):
        return np.einsum("tiab,tjbc,tkcd->tijk", a, b, c)

    want = full(*cores)
    for t in range(count):
        got = full(*(np.asarray(c)[None] for c in out[t].ttv_vec))[0]
        assert np.linalg.norm(got - want[t]) <= 1e-13 * np.linalg.norm(want[t])
