"""Blocks of the element-wise launches: shared among a launch's problems by elements, not by their number."""
import ctypes as C

import pytest

ttcuda = pytest.importorskip("ttcuda")
blocks = ttcuda.lib.ttc_test_elem_blocks
blocks.argtypes = [C.c_longlong, C.c_longlong, C.c_int, C.c_int, C.c_int]
SMS, PER = 148, 1024


@pytest.mark.parametrize("count", [1, 28, 60, 1185, 1680, 2500, 60000])
@pytest.mark.parametrize("n", [1, 900, 5000, 180000, 10 ** 8])
def test_like_problems(count, n):
    """Sixteen blocks per SM over the launch, at least one and no more than there are elements for."""
    b = blocks(n, n * count, PER, count, SMS)
    assert b == max(1, min(16 * SMS // count, -(-n // PER)))


@pytest.mark.parametrize("count", [28, 300, 1185, 2548, 9000])
def test_one_large_problem_among_small_ones(count):
    """The large one gets sixteen blocks at least, whatever the number of the others."""
    n = 500000
    assert blocks(n, n + 50 * (count - 1), PER, count, SMS) == max(16, 16 * SMS // count)


def test_nothing_to_do():
    assert blocks(0, 0, PER, 5, SMS) == 1
