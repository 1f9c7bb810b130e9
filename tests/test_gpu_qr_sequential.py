"""The row-sequential Householder QR at the sizes where its code changes: column steps in registers for each
128 panel rows up to 1024 and in shared memory above, one to three octets of trailing columns per group of
warps, partial last panels, octets and batches, rank-deficient and non-finite inputs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib
P = C.POINTER(C.c_double)
lib.ttc_test_qr_seq.argtypes = [C.c_void_p, C.c_int, C.c_int, P, P, P]


def qr(A):
    m, n = A.shape
    K = min(m, n)
    a, q, r = A.ravel(order="F").copy(), np.empty(m * K), np.empty(K * n)
    ctx = ttcuda.get_context()
    ctx.check(lib.ttc_test_qr_seq(ctx.h, m, n, *(v.ctypes.data_as(P) for v in (a, q, r))))
    return q.reshape((m, K), order="F"), r.reshape((K, n), order="F")


def check(A, Q, R):
    """Each of the K reflectors is orthogonal, and applied, to a few eps of the column norms, and the
    errors of the K steps add up like a random walk: 16 eps sqrt(K)."""
    K = Q.shape[1]
    tol = 16 * np.finfo(float).eps * np.sqrt(K)
    assert np.abs(Q.T @ Q - np.eye(K)).max() <= tol
    assert np.linalg.norm(Q @ R - A) <= tol * np.linalg.norm(A)
    assert not np.tril(R, -1).any()


@pytest.mark.parametrize("m,n", [
    (1, 1), (1, 9), (2, 1), (15, 16), (16, 15), (17, 17), (33, 80), (65, 65), (127, 16), (128, 40), (129, 41), (200, 333),
    (255, 31), (257, 33), (300, 640), (384, 20), (385, 18), (511, 18), (512, 47), (513, 48), (640, 320), (769, 33),
    (897, 17), (1024, 32), (1025, 33), (1039, 17), (1152, 1100), (1536, 24)])
def test_sizes(m, n):
    A = np.random.default_rng(1000 * m + n).standard_normal((m, n))
    check(A, *qr(A))


@pytest.mark.parametrize("m,n", [(40, 30), (300, 70), (700, 40), (1100, 36)])
def test_rank_deficient(m, n):
    """Zero columns, repeated columns and columns that fall off by twelve orders: Q stays orthogonal and Q R
    is A column by column."""
    A = np.random.default_rng(m + n).standard_normal((m, n))
    A[:, 2], A[:, 5] = 0.0, 3.0 * A[:, 1]
    A[:, 6:] *= 10.0 ** -np.linspace(0, 12, n - 6)
    Q, R = qr(A)
    check(A, Q, R)
    tol = 16 * np.finfo(float).eps * np.sqrt(n)
    assert (np.linalg.norm(Q @ R - A, axis=0) <= tol * np.linalg.norm(A, axis=0)).all()


@pytest.mark.parametrize("m,n,at", [(40, 20, (39, 19)), (520, 33, (519, 32)), (1030, 17, (1029, 16))])
def test_non_finite_is_refused(m, n, at):
    A = np.random.default_rng(m).standard_normal((m, n))
    A[at] = np.inf
    with pytest.raises(ttcuda.ArgumentError):
        qr(A)
