"""The Rayleigh gradient's device memory: its two plans share what the first one leaves for the second, so
a context whose workspace an earlier call has grown to any size in between must give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")


def train(g, d, n, r, ops=False):
    rks = [1] + [r] * (d - 1) + [1]
    cores = [np.asfortranarray(g.standard_normal(((n, n) if ops else (n,)) + (rks[k], rks[k + 1])) / np.sqrt(n * rks[k + 1]))
             for k in range(d)]
    return (ttcuda.TToperator if ops else ttcuda.TTvector)(d, cores, (n,) * d, rks)


@pytest.mark.parametrize("d,n,r,R,before", [(32, 2, 132, 8, (117, 118, 119, 120)), (28, 2, 148, 8, (131, 133, 135)),
                                            (30, 3, 76, 14, (67, 68, 69, 70))])
def test_after_a_smaller_gradient(d, n, r, R, before, monkeypatch):
    """At these shapes the second plan (all sites' products in one launch, K split) needs more workspace than
    the first; gradients at the smaller ranks leave workspaces of sizes between the two."""
    g = np.random.default_rng(r)
    H, x = train(g, d, n, R, True), train(g, d, n, r)
    monkeypatch.setattr(ttcuda, "_CTX", ttcuda.Context(0))
    want, Gw = ttcuda.rayleigh_grad(H, x)
    for r0 in before:
        monkeypatch.setattr(ttcuda, "_CTX", ttcuda.Context(0))
        ttcuda.rayleigh_grad(H, train(g, d, n, r0))
        v, G = ttcuda.rayleigh_grad(H, x)
        assert v == want and all(np.array_equal(a, b) for a, b in zip(G, Gw))
