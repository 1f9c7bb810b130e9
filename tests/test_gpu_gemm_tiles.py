"""The grouped FP64 GEMM at the edges of its four output tiles (64 x 64, 64 x 32, 32 x 32, 16 x 16, chosen by
the launch's size), over strides, split dimensions and K splits, and with more problems than one round of the
descriptor search covers."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib
P, PL, PI = C.POINTER(C.c_double), C.POINTER(C.c_longlong), C.POINTER(C.c_int)
lib.ttc_test_gemm_runs.argtypes = [C.c_void_p] + [C.c_int] * 7 + [P, C.c_longlong, PL] * 3 + [C.c_double] * 2 + [C.c_int, PI]
EPS = np.finfo(float).eps


def gemm(m, n, k, batch, m0, n0, k0e, A, ast, B, bst, Cm, cst, beta=0.0):
    ctx, ks, args = ttcuda.get_context(), C.c_int(0), []
    for a, s in ((A, ast), (B, bst), (Cm, cst)):
        args += [a.ctypes.data_as(P), a.size, np.asarray(s, dtype=np.int64).ctypes.data_as(PL)]
    ctx.check(lib.ttc_test_gemm_runs(ctx.h, m, n, k, batch, m0, n0, k0e, *args, 1.0, beta, 1, C.byref(ks)))
    return ks.value


def check(got, a, b, c0):
    """k products and additions (and the old value): an element is off by (k + 2) eps of the sum of the
    magnitudes at most."""
    want, mag = a @ b + c0, np.abs(a) @ np.abs(b) + np.abs(c0)
    assert (np.abs(got - want) <= (a.shape[-1] + 2) * EPS * mag).all()


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (15, 17, 16), (16, 16, 33), (17, 15, 8), (31, 33, 15), (32, 32, 16), (33, 31, 17), (63, 65, 48), (64, 64, 64),
                                   (65, 63, 4), (97, 40, 80), (129, 95, 31)])
@pytest.mark.parametrize("trans", [False, True])
def test_tiles_agree(m, n, k, trans):
    """One product alone and as a batch of 40, 160 and 700: the tile changes with the number of output
    tiles in the launch, no bit of the result does."""
    g = np.random.default_rng(m * n + k)
    batch = 700
    a, b = g.standard_normal((batch, m, k)), g.standard_normal((batch, k, n))
    A = (a if trans else a.transpose(0, 2, 1)).copy().ravel()
    B = (b if trans else b.transpose(0, 2, 1)).copy().ravel()
    ast = [k, 0, 1, 0, m * k] if trans else [1, 0, m, 0, m * k]
    bst = [n, 0, 1, 0, n * k] if trans else [1, 0, k, 0, n * k]
    cst = [n, 0, 1, 0, m * n] if trans else [1, 0, m, 0, m * n]
    out = []
    for nb in (1, 40, 160, 700):
        Cm = np.full(nb * m * n, np.nan)
        assert gemm(m, n, k, nb, m, n, k, A[:nb * m * k], ast, B[:nb * n * k], bst, Cm, cst) == 1
        out.append(Cm.reshape(nb, m * n))
    for o in out[:-1]:
        assert np.array_equal(o, out[-1][:len(o)])
    c = out[-1].reshape(batch, m, n) if trans else out[-1].reshape(batch, n, m).transpose(0, 2, 1)
    check(c, a, b, np.zeros_like(c))


@pytest.mark.parametrize("m,n,k,k0e,batch", [(33, 30, 40, 5, 1), (66, 70, 55, 11, 90), (64, 96, 1050, 7, 1),
                                             (40, 66, 1300, 13, 3), (70, 33, 3000, 3, 2)])
def test_split_dimensions(m, n, k, k0e, batch):
    """Rows, columns and K each split over two strides, with and without K splits (k above 1024), and
    added to the old C."""
    g = np.random.default_rng(k)
    m0, n0 = (m + 2) // 3, (n + 1) // 2
    a, b = g.standard_normal((batch, m, k)), g.standard_normal((batch, k, n))
    c0 = g.standard_normal((batch, m, n))
    i, j, kk = np.arange(m), np.arange(n), np.arange(k)

    def place(x, r, r0, rs, c, c_0, cs):
        """x in a buffer at (r % r0) rs[0] + (r // r0) rs[1] + (c % c_0) cs[0] + (c // c_0) cs[1]."""
        at = ((r % r0) * rs[0] + (r // r0) * rs[1])[:, None] + ((c % c_0) * cs[0] + (c // c_0) * cs[1])[None, :]
        last = (r0 - 1) * rs[0] + r[-1] // r0 * rs[1] + (c_0 - 1) * cs[0] + c[-1] // c_0 * cs[1]   # of whole blocks
        size = int(last) + 3
        buf = np.zeros((batch, size))
        buf[:, at.ravel()] = x.reshape(batch, -1)
        return buf.ravel().copy(), size, at

    nk = (k + k0e - 1) // k0e
    A, a_b, _ = place(a, i, m0, (1, m0 * k), kk, k0e, (m0, m0 * k0e))
    B, b_b, _ = place(b, kk, k0e, (n0 * nk, n0), j, n0, (1, n0 * nk * k0e))
    Cm, c_b, at = place(c0, i, m0, (n0, m0 * n0), j, n0, (1, m0 * n0 * 3))
    ks = gemm(m, n, k, batch, m0, n0, k0e, A, [1, m0 * k, m0, m0 * k0e, a_b],
              B, [n0 * nk, n0, 1, n0 * nk * k0e, b_b], Cm, [n0, m0 * n0, 1, m0 * n0 * 3, c_b], beta=1.0)
    assert (ks > 1) == (k > 1024)
    check(Cm.reshape(batch, -1)[:, at.ravel()].reshape(batch, m, n), a, b, c0)


def test_many_problems():
    """70 trains of ranks 1 to 6 rounded together at tolerance 0: every contraction of the sweep is one
    launch of up to 70 problems, and each train is again the tensor that it was (a few eps per step)."""
    g = np.random.default_rng(0)
    dims, tts = (3, 4, 2, 3), []
    for t in range(70):
        r = [1, 1 + t % 3, 1 + t % 6, 1 + t % 2, 1]
        tts.append([g.standard_normal((dims[q], r[q], r[q + 1])) for q in range(4)])

    def full(cores):
        x = np.ones((1, 1))
        for c in cores:
            x = np.einsum("ia,xab->ixb", x, c).reshape(-1, c.shape[2])
        return x.ravel()

    vec = [ttcuda.TTvector(4, [np.asfortranarray(c) for c in t], dims, [1] + [c.shape[2] for c in t]) for t in tts]
    xb = ttcuda.DeviceBatch.from_tts(vec)
    yb = ttcuda.DeviceBatch(dims, [v.ttv_rks for v in vec])
    xb.round_det(yb, tol=0.0)
    for t, y in zip(tts, yb.download()):
        want = full(t)
        assert np.linalg.norm(full(y.ttv_vec) - want) <= 1e-13 * np.linalg.norm(want)
