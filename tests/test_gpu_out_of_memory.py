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
