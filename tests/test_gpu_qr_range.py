"""Householder QR of columns whose squares leave the range of FP64."""
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


def tolerance(K):
    """Each of the K reflectors is orthogonal, and applied, to a few eps of the column norms, and the errors of
    the K steps add up like a random walk: 16 eps sqrt(K)."""
    return 16 * np.finfo(float).eps * np.sqrt(K)


# below 1e-154 and above 1e154 the squared norm of a column is no normal number; R's smallest entries have
# to stay normal numbers themselves
@pytest.mark.parametrize("m,n", [(16, 5), (97, 35), (200, 40), (300, 20), (700, 18), (1200, 17)])
@pytest.mark.parametrize("e", [-980, -600, -520, -512, -505, 450, 505, 520, 1000])
def test_scaled(m, n, e):
    """A power of two leaves every digit of Q and R as it was."""
    A = np.random.default_rng(m).standard_normal((m, n))
    Q, R = qr(A)
    assert np.abs(Q.T @ Q - np.eye(n)).max() <= tolerance(n)
    assert np.linalg.norm(Q @ R - A) <= tolerance(n) * np.linalg.norm(A)
    Qs, Rs = qr(np.ldexp(A, e))
    assert np.array_equal(Qs, Q) and np.array_equal(Rs, np.ldexp(R, e))


@pytest.mark.parametrize("m,n", [(60, 40), (300, 33), (600, 33)])
def test_columns_of_different_size(m, n):
    """Columns from 2^-520 to 1 beside one another: every column of Q R is A's to the column's own accuracy."""
    B = np.random.default_rng(n).standard_normal((m, n))
    e = np.zeros(n, int)
    e[3::5], e[4::7] = -520, -300
    Q, R = qr(np.ldexp(B, e))
    assert np.abs(Q.T @ Q - np.eye(n)).max() <= tolerance(n)
    assert (np.linalg.norm(Q @ np.ldexp(R, -e) - B, axis=0) <= tolerance(n) * np.linalg.norm(B, axis=0)).all()


@pytest.mark.parametrize("scale", [1e-157, 1e-170, 1e160])
def test_orthogonalize(scale):
    """A train one of whose cores has entries of that size is the same tensor afterwards."""
    g = np.random.default_rng(11)
    dims, r = (3, 4, 3, 2), [1, 3, 9, 2, 1]
    cores = [np.asfortranarray(g.standard_normal((n, r[k], r[k + 1]))) for k, n in enumerate(dims)]
    cores[1] *= scale
    x = ttcuda.TTvector(4, cores, dims, r)

    def full(t):
        return np.einsum("iab,jbc,kcd,lde->ijkl", *(np.asarray(c) for c in t.ttv_vec))

    want = full(x)
    for i in (1, 2, 4):
        got = full(ttcuda.orthogonalize(x, i))
        assert np.linalg.norm((got - want) / scale) <= 1e-13 * np.linalg.norm(want / scale)
