"""The gradient's two environment chains, run side by side, over lengths where they do not meet in step (one
site, two, odd counts) and over ragged dimensions and ranks, in both precisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
from oracle import tt_oracle as o  # noqa: E402


@pytest.mark.parametrize("precision,eps", [("fp64", 2.0 ** -53), ("fp32", 2.0 ** -24)])
@pytest.mark.parametrize("dims,r,R", [((3,), [1, 1], [1, 1]), ((2, 5), [1, 2, 1], [1, 4, 1]),
                                      ((4, 2, 3), [1, 3, 7, 1], [1, 2, 5, 1]),
                                      ((2, 3, 2, 4, 2), [1, 2, 33, 40, 2, 1], [1, 4, 1, 17, 3, 1]),
                                      ((3, 2) * 4, [1, 3, 6, 35, 70, 66, 5, 3, 1], [1, 2, 3, 9, 4, 7, 3, 2, 1])])
def test_against_oracle(dims, r, R, precision, eps):
    """Positive cores and a positive symmetric operator: every sum is of one sign, so a product of sums is off
    by at most the sum of their lengths times eps of itself.  The gradient is 2 (Heff x - R Neff x) / <x|x>,
    two such quantities, of together |G| + 4 R Neff x / <x|x>."""
    g = np.random.default_rng(len(dims))
    d = len(dims)
    cores = [np.asfortranarray(g.uniform(0.1, 1.0, (n, r[k], r[k + 1]))) for k, n in enumerate(dims)]
    ops = []
    for k, n in enumerate(dims):
        c = g.uniform(0.1, 1.0, (n, n, R[k], R[k + 1]))
        ops.append(np.asfortranarray(0.5 * (c + c.transpose(1, 0, 2, 3))))
    want, Gw = o.rayleigh_value_and_grad(o.TToperator(d, ops, dims, R, [0] * d), o.TTvector(d, cores, dims, r, [0] * d))
    x = ttcuda.TTvector(d, cores, dims, r)
    v, G = ttcuda.rayleigh_grad(ttcuda.TToperator(d, ops, dims, R), x, precision=precision)
    nn = ttcuda.dot(x, x)
    lengths = sum(2 * r[k + 1] + n * R[k + 1] + n * r[k + 1] + n * r[k] + R[k] * r[k] for k, n in enumerate(dims))
    tol = 4 * (lengths + 8) * eps
    assert abs(v - want) <= tol * want
    for k, (a, b) in enumerate(zip(G, Gw)):
        assert a.shape == b.shape
        assert (np.abs(a - b) <= tol * (np.abs(b) + 4 * want / nn * neff(cores, k))).all()


def neff(cores, k):
    """Neff_k x_k by full contraction of the norm network on both sides."""
    left, right = np.ones((1, 1)), np.ones((1, 1))
    for c in cores[:k]:
        left = np.einsum("ac,iab,icd->bd", left, c, c)
    for c in reversed(cores[k + 1:]):
        right = np.einsum("bd,iab,icd->ac", right, c, c)
    return np.einsum("ac,icd,bd->iab", left, cores[k], right)
