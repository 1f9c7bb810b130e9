"""Calls that meet the end of the device's memory (a status that the allocation attempts are told to return; no
memory is filled): an error, nothing lost, and the next call works."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ttcuda = pytest.importorskip("ttcuda")
lib = ttcuda.lib


def train(r, d=8):
    g = np.random.default_rng(r)
    rks = [1] + [r] * (d - 1) + [1]
    return ttcuda.TTvector(d, [np.asfortranarray(g.standard_normal((2, rks[k], rks[k + 1])) / np.sqrt(2 * r)) for k in range(d)],
                           (2,) * d, rks)


def blocks(ctx):
    idle, used = C.c_longlong(), C.c_int()
    ctx.check(lib.ttc_test_blocks(ctx.h, C.byref(idle), C.byref(used)))
    return idle.value, used.value


@pytest.mark.parametrize("after", [0, 1, 2, 3, 4])
def test_failed_call_gives_its_blocks_back(after, monkeypatch):
    """Both attempts of one allocation fail, each of a call's allocations in turn: the blocks that the call had
    taken by then are idle or freed again."""
    ctx = ttcuda.Context(0)
    monkeypatch.setattr(ttcuda, "_CTX", ctx)
    x, y = train(300), train(310)
    want = ttcuda.dot(x, y)
    in_use = blocks(ctx)[1]
    ctx.check(lib.ttc_test_fail_alloc(ctx.h, after, 2))
    with pytest.raises(Exception, match="TTC_ENOMEM|out of memory"):
        ttcuda.dot(train(350), train(360))
    ctx.check(lib.ttc_test_fail_alloc(ctx.h, 0, 0))
    assert blocks(ctx)[1] == in_use
    assert ttcuda.dot(x, y) == want


def idle_context(monkeypatch, ranks=(300,)):
    ctx = ttcuda.Context(0)
    monkeypatch.setattr(ttcuda, "_CTX", ctx)
    for r in ranks:
        ttcuda.dot(train(r), train(r + 10))
    assert blocks(ctx)[0] > 0
    return ctx


def test_idle_blocks_of_every_context_go_when_memory_runs_out(monkeypatch):
    """One attempt of another context to allocate fails: the call succeeds at the second one, and no context of
    the device holds an idle block from before it."""
    a, b, c = idle_context(monkeypatch), idle_context(monkeypatch), idle_context(monkeypatch)
    x, y = train(500), train(510)                      # larger than any idle block
    c.check(lib.ttc_test_fail_alloc(c.h, 0, 1))
    got = ttcuda.dot(x, y)
    assert blocks(a) == (0, 0) and blocks(b) == (0, 0)
    assert got == ttcuda.dot(x, y)


def test_trim(monkeypatch):
    ctx = idle_context(monkeypatch)
    ctx.trim()
    assert blocks(ctx) == (0, 0)
    assert np.isfinite(ttcuda.dot(train(300), train(310)))


def test_idle_blocks_stay_within_their_bound(monkeypatch):
    """0.8 GB of operands of growing size, none of which fits a block that is idle."""
    ctx = idle_context(monkeypatch, range(300, 1000, 70))
    assert blocks(ctx)[0] <= 512 << 20


def test_blocks_below_a_megabyte_are_kept(monkeypatch):
    """Two operands of 213 KB: left to the driver, they may be the last of a slab, which each call then maps and
    unmaps."""
    ctx = ttcuda.Context(0)
    monkeypatch.setattr(ttcuda, "_CTX", ctx)
    x = train(48, 16)
    size = sum(c.nbytes for c in x.ttv_vec)
    assert 100 << 10 < size < 1 << 20
    ttcuda.dot(x, x)
    assert blocks(ctx)[0] >= 2 * size and blocks(ctx)[1] == 0
    for r in range(8, 200, 2):
        ttcuda.norm(train(r, 4))
    held = blocks(ctx)[0]
    ctx.trim()
    assert 0 < held <= 512 << 20 and blocks(ctx) == (0, 0)
