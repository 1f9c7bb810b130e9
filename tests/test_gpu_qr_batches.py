"""Householder QRs of many problems in one launch, as the batched roundings issue them: the eight-warp kernel at
257 to 512 rows (which only launches of more than 18 problems reach), clusters of eight CTAs to one, bounds
read from the device, and the non-finite report.  The row-sequential kernel keeps its bits in all of them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
P = C.POINTER(C.c_double)


def qr(A, mb=-1, nb=-1, mult=1, sequential=False, tall=0):
    """A: (count, n, m), each matrix column by column.  Q (count, K, m) and R (count, n, K) alike."""
    count, n, m = A.shape
    K = min(m, n)
    A = np.ascontiguousarray(A)
    Q, R = np.empty((count, K, m)), np.empty((count, n, K))
    ctx = ttcuda.get_context()
    ctx.check(ttcuda.lib.ttc_test_qr_many(ctx.h, count, m, n, *(v.ctypes.data_as(P) for v in (A, Q, R)), mb, nb, mult,
                                          int(sequential), tall))
    return Q, R


def check(A, Q, R):
    """Each of the K reflectors is orthogonal, and applied, to a few eps of the column norms, and the errors of
    the K steps add up like a random walk: 16 eps sqrt(K)."""
    K = Q.shape[1]
    tol = 16 * np.finfo(float).eps * np.sqrt(K)
    assert np.abs(Q @ Q.transpose(0, 2, 1) - np.eye(K)).max() <= tol
    err = np.linalg.norm(R @ Q - A, axis=(1, 2))
    assert (err <= tol * np.linalg.norm(A, axis=(1, 2))).all()
    assert not np.triu(R, 1).any()                     # R^T row by row


@pytest.mark.parametrize("m,n", [(130, 24), (257, 40), (300, 33), (400, 24), (511, 17), (512, 48), (300, 310)])
def test_many_problems(m, n):
    """20, 40, 80 and 160 problems (clusters of 8, 4, 2 and 1): the same bits in each."""
    A = np.random.default_rng(m * n).standard_normal((160, n, m))
    Q, R = qr(A)
    check(A, Q, R)
    for count in (20, 40, 80):
        q, r = qr(A[:count])
        assert np.array_equal(q, Q[:count]) and np.array_equal(r, R[:count])


@pytest.mark.parametrize("count", [1, 20, 160])
@pytest.mark.parametrize("m,n,mb,nb,mult", [(400, 64, 300, 50, 1), (512, 40, 129, 20, 2), (300, 96, 40, 96, 1), (300, 40, 0, 40, 1),
                                            (512, 90, 512, 0, 1), (140, 70, 17, 16, 2)])
def test_device_bounds(count, m, n, mb, nb, mult):
    A = np.random.default_rng(m + n).standard_normal((count, n, m))
    A[:, nb * mult:] = 0.0
    A[:, :, mb * mult:] = 0.0
    check(A, *qr(A, mb, nb, mult))


@pytest.mark.parametrize("count,m,n", [(1, 40, 20), (1, 520, 33), (1, 1030, 17), (20, 257, 20), (30, 500, 33), (30, 60, 17)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_is_refused(count, m, n, value):
    """The first entry of the first problem, one amid a column, the last one of the last panel."""
    A = np.random.default_rng(m).standard_normal((count, n, m))
    for at in ((0, 0, 0), (count // 2, n // 2, m // 2 + 1), (count - 1, n - 1, m - 1)):
        B = A.copy()
        B[at] = value
        with pytest.raises(ttcuda.ArgumentError):
            qr(B)


@pytest.mark.parametrize("m,n", [(130, 64), (276, 138), (700, 100), (1100, 40)])
def test_sequential_bits(m, n):
    """One matrix alone (a cluster of eight CTAs) and among 40, 100 and 250 (four, two, one), beside a taller
    one: the same bits."""
    A = np.random.default_rng(m).standard_normal((1, n, m)) * np.logspace(0, -9, n)[None, :, None]
    Q, R = qr(A, sequential=True)
    check(A, Q, R)
    for count, tall in ((1, 1536), (40, 0), (100, 1300), (250, 0)):
        q, r = qr(np.repeat(A, count, axis=0), sequential=True, tall=tall)
        assert (q == Q).all() and (r == R).all()
