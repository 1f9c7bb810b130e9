"""Output tiles of the grouped FP64 GEMM by the size of the launch (0: 64 x 64, 1: 64 x 32, 2: 32 x 32, 3: 16 x 16)."""
import ctypes as C

import pytest

ttcuda = pytest.importorskip("ttcuda")
pick = ttcuda.lib.ttc_test_gemm_tile
pick.argtypes = [C.c_int] * 6
SMS = 148


@pytest.mark.parametrize("m,n,count", [(700, 700, 1), (1000, 60, 8), (100, 50, 60), (256, 256, 8), (768, 768, 1), (1100, 500, 1)])
def test_no_large_tile_alone_on_its_sm(m, n, count):
    """112 to 148 tiles of 64 x 64: one per SM, whose four warps leave its tensor cores idle half the time."""
    assert -(-m // 64) * -(-n // 64) * count <= SMS
    assert pick(m, n, 300, 1, count, SMS) == 1


@pytest.mark.parametrize("m,n,count", [(10, 5, 1), (30, 15, 1), (64, 64, 3), (138, 138, 1)])
def test_few_outputs_take_the_smallest(m, n, count):
    assert pick(m, n, 100, 1, count, SMS) == 3


@pytest.mark.parametrize("m,n,count", [(960, 960, 1), (256, 2048, 2), (4096, 4096, 1), (1280, 1280, 1)])
def test_full_turns_take_the_largest(m, n, count):
    assert pick(m, n, 256, 1, count, SMS) == 0
