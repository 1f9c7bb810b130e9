"""The Rayleigh gradient's device memory.  Its two plans share what the first one leaves for the second, so
a context whose workspace an earlier call has grown to any size in between must give the same bits; and above
a bound it keeps only every ckpt_every-th left environment."""
import ctypes as C

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


def grad_keep(ctx, nbytes):
    ws = C.c_longlong()
    ctx.check(ttcuda.lib.ttc_test_grad_keep(ctx.h, C.c_longlong(nbytes), C.byref(ws)))
    return ws.value


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("d", [1, 2, 9, 12])
def test_checkpointed_gradient(d, precision, monkeypatch):
    """Below 512 terms no sum is split, and a recomputed environment is the same bits: so is the gradient,
    for segments of one site, that end short, and of more sites than there are."""
    g = np.random.default_rng(d)
    H, x = train(g, d, 3, 5, True), train(g, d, 3, 21)
    want, Gw = ttcuda.rayleigh_grad(H, x, precision=precision)
    ctx = ttcuda.Context(0)
    monkeypatch.setattr(ttcuda, "_CTX", ctx)
    grad_keep(ctx, 0)
    for ckpt in (2, 3, 4, 5, 8, 20, 1, 0):
        v, G = ttcuda.rayleigh_grad(H, x, ckpt_every=ckpt, precision=precision)
        assert v == want and all(np.array_equal(a, b) for a, b in zip(G, Gw))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_checkpoints_bound_the_memory(precision, monkeypatch):
    """Of 48 sites, each with an environment of r r R numbers and products of n r r R (n = 2): with all kept
    48 x 3 such blocks; with every sixth environment kept 8 + 5 environments and the products of six sites, 25
    blocks, and in both the scratch of a turn, at most 8."""
    g = np.random.default_rng(1)
    H, x = train(g, 48, 2, 6, True), train(g, 48, 2, 64)
    used = {}
    for keep, ckpt in ((1 << 40, 6), (0, 1), (0, 6)):
        ctx = ttcuda.Context(0)
        monkeypatch.setattr(ttcuda, "_CTX", ctx)
        grad_keep(ctx, keep)
        ttcuda.rayleigh_grad(H, x, ckpt_every=ckpt, precision=precision)
        used[keep, ckpt] = grad_keep(ctx, keep)
    assert used[0, 1] == used[1 << 40, 6]
    assert used[0, 6] <= 0.4 * used[0, 1]
