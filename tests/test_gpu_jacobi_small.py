"""The one-warp Jacobi SVD (up to 32 rows and columns) at the edges of its two widths (16 and 32), odd and
even column counts, rectangular, rank-deficient and zero inputs."""
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
    x, s, perm, sw = A.ravel(order="F").copy(), np.empty(n), np.empty(n, np.int32), C.c_int(0)
    ctx = ttcuda.get_context()
    ctx.check(lib.ttc_test_jacobi(ctx.h, m, n, x.ctypes.data_as(P), 0, None, s.ctypes.data_as(P), perm.ctypes.data_as(PI),
                                  C.byref(sw)))
    return x.reshape((m, n), order="F"), s, perm, sw.value


def check(A):
    """X = A V with V orthogonal: X X^T is A A^T up to 4 eps for each of a column's at most 12 n rotations.
    Columns of X are left at max(m, 16) eps of orthogonal, or below that part of ||A||_F, where they count as
    zero; the singular values, the norms of X's columns, are off by what that leaves, sqrt(n) of it."""
    m, n = A.shape
    X, s, perm, sweeps = jacobi(A)
    fro, tol = np.linalg.norm(A), max(m, 16) * EPS
    assert 0 < sweeps <= 12
    assert np.abs(X @ X.T - A @ A.T).max() <= 48 * n * EPS * fro ** 2
    d = np.linalg.norm(X, axis=0)
    assert np.abs(s - d).max() <= 4 * EPS * max(m, 1) * fro
    assert sorted(perm) == list(range(n)) and (np.diff(s[perm]) <= 0).all()
    want = np.zeros(n)
    want[:min(m, n)] = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s[perm] - want).max() <= (2 * tol * np.sqrt(n) + 48 * n * EPS) * fro


@pytest.mark.parametrize("m,n", [(1, 1), (1, 2), (2, 1), (2, 2), (3, 2), (3, 3), (7, 8), (8, 7), (15, 15), (15, 16), (16, 16),
                                 (16, 17), (17, 16), (17, 17), (9, 31), (31, 9), (31, 32), (32, 31), (32, 32), (33, 32)])
def test_sizes(m, n):
    check(np.random.default_rng(100 * m + n).standard_normal((m, n)))


@pytest.mark.parametrize("n", [2, 9, 16, 24, 32])
def test_graded_and_deficient(n):
    g = np.random.default_rng(n)
    check(np.triu(g.standard_normal((n, n))) * 10.0 ** -np.linspace(0, 14, n))
    A = g.standard_normal((n, max(1, n // 2))) @ g.standard_normal((max(1, n // 2), n))
    A[:, n // 2] = 0.0
    check(A)


@pytest.mark.parametrize("n", [1, 16, 31])
def test_zero(n):
    X, s, perm, _ = jacobi(np.zeros((n, n)))
    assert not X.any() and not s.any() and sorted(perm) == list(range(n))
