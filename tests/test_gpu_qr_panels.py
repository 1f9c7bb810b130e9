"""Householder QR kernel at the sizes where its panel code changes: the register widths (64, 128, 256,
512 and 1024 panel rows), the eight- and sixteen-warp kernels, partial last panels and octets, odd
leading dimensions (no 16-byte loads) and rank-deficient inputs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib
P = C.POINTER(C.c_double)
lib.ttc_test_qr.argtypes = [C.c_void_p, C.c_int, C.c_int, P, P, P]


def qr(A):
    m, n = A.shape
    K = min(m, n)
    a, q, r = A.ravel(order="F").copy(), np.empty(m * K), np.empty(K * n)
    ctx = ttcuda.get_context()
    ctx.check(lib.ttc_test_qr(ctx.h, m, n, *(v.ctypes.data_as(P) for v in (a, q, r))))
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
    (1, 1), (1, 9), (2, 1), (7, 7), (8, 16), (15, 16), (16, 15), (17, 17), (33, 80), (63, 17), (64, 33), (65, 65),
    (80, 64), (127, 16), (128, 40), (129, 41), (200, 333), (255, 100), (256, 31), (257, 33), (271, 129), (511, 18),
    (512, 47), (513, 48), (527, 24), (640, 50), (769, 33), (1023, 20), (1024, 32), (1025, 33), (1039, 17), (1536, 24)])
def test_qr_sizes(m, n):
    A = np.random.default_rng(1000 * m + n).standard_normal((m, n))
    Q, R = qr(A)
    check(A, Q, R)
    # the reflectors' sign convention is LAPACK's (beta = -sign(alpha) ||x||); the last diagonal
    # entry of a square matrix has no reflector to fix it beyond rounding
    d = np.sign(np.diag(np.linalg.qr(A)[1]))
    assert np.array_equal(np.sign(np.diag(R)), d)


@pytest.mark.parametrize("m,n,rank", [(40, 20, 0), (100, 48, 7), (130, 64, 33), (301, 65, 16), (600, 40, 12)])
def test_qr_rank_deficient(m, n, rank):
    g = np.random.default_rng(m + n)
    A = g.standard_normal((m, rank)) @ g.standard_normal((rank, n)) if rank else np.zeros((m, n))
    A[:, n // 3] = 0.0                                # an exactly zero column among them
    check(A, *qr(A))


@pytest.mark.parametrize("scale", [1e-150, 1e-30, 1e140])
def test_qr_scaled(scale):
    A = scale * np.random.default_rng(3).standard_normal((97, 35))
    check(A, *qr(A))
