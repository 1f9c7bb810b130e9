"""Gram-block Jacobi SVD kernel at the sizes where its blocks change: one to many 16-column blocks, odd
block counts, partial blocks, rows that are not multiples of 4 or 8, odd leading dimensions (no
16-byte copies), and the same bits on every run."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib
P, PI = C.POINTER(C.c_double), C.POINTER(C.c_int)
lib.ttc_test_jacobi.argtypes = [C.c_void_p, C.c_int, C.c_int, P, C.c_int, P, P, PI, PI]
EPS = np.finfo(float).eps


def jacobi(A):
    m, n = A.shape
    x, s, w = A.ravel(order="F").copy(), np.empty(n), np.empty(1)
    perm, info = np.zeros(n, dtype=np.int32), np.zeros(1, dtype=np.int32)
    ctx = ttcuda.get_context()
    ctx.check(lib.ttc_test_jacobi(ctx.h, m, n, x.ctypes.data_as(P), 0, w.ctypes.data_as(P), s.ctypes.data_as(P),
                                  perm.ctypes.data_as(PI), info.ctypes.data_as(PI)))
    assert info[0] > 0
    return x.reshape((m, n), order="F"), s, perm


def check(A, X, s, perm):
    m, n = A.shape
    ref = np.linalg.svd(A, compute_uv=False)
    # a column takes part in about 10 n rotations, each a few eps off: a random walk
    tol = 8 * EPS * np.sqrt(10 * n)
    assert sorted(perm.tolist()) == list(range(n))
    assert np.all(np.diff(s[perm]) <= 0)
    assert np.abs(s[perm] - ref).max() <= tol * max(ref[0], 1e-300)
    assert np.linalg.norm(X @ X.T - A @ A.T) <= 2 * tol * np.linalg.norm(A) ** 2   # X = A W, W orthogonal
    big = s > max(m, 16) * EPS * np.linalg.norm(A)      # the kernel's zero threshold
    if big.any():
        U = X[:, big] / s[big]
        off = U.T @ U - np.eye(U.shape[1])
        # pairs pass the rotation test below max(m, 16) eps, measured to another such error
        assert np.abs(off).max() <= 2 * max(m, 16) * EPS


@pytest.mark.parametrize("m,n", [
    (33, 17), (33, 33), (34, 32), (40, 35), (47, 47), (48, 48), (49, 49), (63, 63), (64, 64), (65, 65), (79, 70),
    (96, 96), (111, 111), (127, 127), (129, 129), (145, 140), (200, 200), (255, 255), (257, 257), (300, 290), (511, 100)])
def test_jacobi_sizes(m, n):
    g = np.random.default_rng(1000 * m + n)
    A = g.standard_normal((m, n)) * 10.0 ** (-3.0 * np.arange(n) / n)
    A = np.linalg.qr(np.linalg.qr(A, mode="r").T, mode="r").T if m >= n else A     # the preconditioned factor
    if m > A.shape[0]:
        A = np.vstack([A, np.zeros((m - A.shape[0], n))]) + 0.0
    X, s, perm = jacobi(A)
    check(A, X, s, perm)
    for _ in range(2):
        X2, s2, perm2 = jacobi(A)
        assert np.array_equal(X, X2) and np.array_equal(s, s2) and np.array_equal(perm, perm2)


@pytest.mark.parametrize("scale", [1e-120, 1e120])
def test_jacobi_scaled(scale):
    A = scale * np.random.default_rng(5).standard_normal((70, 60))
    X, s, perm = jacobi(A)
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s[perm] - ref).max() <= 8 * EPS * np.sqrt(600) * ref[0]
