"""One-shot calls whose operands live in device blocks kept between calls: what an earlier call of another
shape left in a block must not be seen, and the blocks go with their context."""
import numpy as np
import pytest

import torch

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")


def train(g, dims, r, ops=False):
    d = len(dims)
    rks = [1] + [r] * (d - 1) + [1]
    cores = [np.asfortranarray(g.standard_normal(((n, n) if ops else (n,)) + (rks[k], rks[k + 1])) / np.sqrt(n * rks[k + 1]))
             for k, n in enumerate(dims)]
    return (ttcuda.TToperator if ops else ttcuda.TTvector)(d, cores, dims, rks)


def calls(x, y, H):
    """apply, dot, partial contraction, both gradients, addition, norm: every kind of operand and result."""
    out = [np.asarray(c) for c in ttcuda.mpo_apply(H, x).ttv_vec]
    out += [np.asarray(ttcuda.dot(x, y)), np.asarray(ttcuda.dot_operator(x, H, y))]
    out += [np.asarray(w) for w in ttcuda.partial_contraction(x, y)]
    for precision in ("fp64", "fp32"):
        v, grads = ttcuda.rayleigh_grad(H, x, ckpt_every=2, precision=precision)
        out += [np.asarray(v)] + [np.asarray(c) for c in grads]
    return out + [np.asarray(c) for c in ttcuda.tt_add(x, y).ttv_vec] + [np.asarray(ttcuda.norm(x))]


def test_blocks_carry_nothing_over(monkeypatch):
    """Three shapes (blocks from 0.3 to 40 MB) in turn, each one's results bit for bit those of a fresh
    context, whatever ran before it."""
    g = np.random.default_rng(5)
    shapes = [((2, 3, 2, 2, 3, 2), 150, 90, 6), ((3, 2, 4, 2), 61, 200, 3), ((2,) * 8, 200, 120, 9)]
    cases = [(train(g, n, r), train(g, n, s), train(g, n, R, True)) for n, r, s, R in shapes]
    fresh = []
    for c in cases:
        monkeypatch.setattr(ttcuda, "_CTX", ttcuda.Context(0))
        fresh.append(calls(*c))
    monkeypatch.setattr(ttcuda, "_CTX", ttcuda.Context(0))
    for i in (0, 1, 2, 0, 2, 1, 1, 0):
        got = calls(*cases[i])
        assert len(got) == len(fresh[i]) and all(np.array_equal(a, b) for a, b in zip(got, fresh[i]))


def test_gradient_layout():
    """The gradient's cores in the caller's layout: the directional derivative of the quotient along a random
    train of the same ranks, by central differences (error h^2 times the third derivative plus eps / h)."""
    g = np.random.default_rng(6)
    dims = (2, 3, 4, 2)
    x, H = train(g, dims, 5), train(g, dims, 3, True)
    for k, n in enumerate(dims):                       # a symmetric operator
        c = H.tto_vec[k]
        H.tto_vec[k] = np.asfortranarray(0.5 * (c + c.transpose(1, 0, 2, 3)))
    v = train(g, dims, 5)

    def quotient(t):
        y = ttcuda.TTvector(4, [np.asfortranarray(a + t * b) for a, b in zip(x.ttv_vec, v.ttv_vec)], dims, x.ttv_rks)
        return ttcuda.dot_operator(y, H, y) / ttcuda.dot(y, y)

    val, grads = ttcuda.rayleigh_grad(H, x, ckpt_every=1)
    assert abs(val - quotient(0.0)) <= 1e-13 * max(1.0, abs(val))
    h = 1e-4
    slope = sum(float(np.vdot(a, b)) for a, b in zip(grads, v.ttv_vec))
    assert abs(slope - (quotient(h) - quotient(-h)) / (2 * h)) <= 1e-5 * max(1.0, abs(slope))


def test_blocks_are_given_back(monkeypatch):
    """A context holds no more than its bound of idle blocks (512 MiB) and nothing once it is gone."""
    g = np.random.default_rng(7)
    keep = ttcuda.get_context()
    torch.cuda.synchronize()
    ctx = ttcuda.Context(0)
    monkeypatch.setattr(ttcuda, "_CTX", ctx)
    x, H = train(g, (2,) * 6, 40), train(g, (2,) * 6, 3, True)
    ttcuda.mpo_apply(H, x)
    before = torch.cuda.mem_get_info()[0]
    for r in (100, 300, 180, 260, 140, 340, 220):
        ttcuda.norm(train(g, (2,) * 10, r))
        ttcuda.tt_add(train(g, (2,) * 10, r), train(g, (2,) * 10, r + 7))
    held = before - torch.cuda.mem_get_info()[0]
    monkeypatch.setattr(ttcuda, "_CTX", keep)
    ctx.close()
    after = torch.cuda.mem_get_info()[0]
    assert held > 0 and after >= before - (4 << 20)
