"""The rule that cuts K into parts, on the CPU: where the partial sums go in a scratch at any address."""
import ctypes

import pytest


def rule(rows, cols, k, address, size):
    from dlprimitives_b200 import capi
    parts, wanted, offset = ctypes.c_int(), ctypes.c_size_t(), ctypes.c_size_t()
    capi.check(capi.lib().dlp_split_rule(rows, cols, k, address, size, ctypes.byref(parts), ctypes.byref(wanted), ctypes.byref(offset)))
    return parts.value, wanted.value, offset.value


# InnerProduct heads, 3x3 layers over 7x7 and 14x14 planes, a ragged product
SHAPES = [(1, 1000, 2048), (128, 1000, 2048), (49, 512, 4608), (196, 256, 2304), (300, 33, 1001)]


@pytest.mark.parametrize("rows,cols,k", SHAPES)
@pytest.mark.parametrize("shift", range(0, 17))
def test_partial_sums_are_aligned(rows, cols, k, shift):
    """They are read 16 bytes at a time, wherever the caller's scratch starts, and the bytes that a plan asks for are enough for that."""
    base = 1 << 20
    parts, wanted, _ = rule(rows, cols, k, base, 1 << 40)
    assert parts > 1
    got, _, offset = rule(rows, cols, k, base + shift, wanted)
    assert got == parts
    assert (base + shift + offset) % 16 == 0
    columns = -(-cols // (32 if cols <= 32 else 64 if cols <= 64 else 128)) * (32 if cols <= 32 else 64 if cols <= 64 else 128)
    assert offset + got * (-(-rows // 128) * 128) * columns * 4 <= wanted


@pytest.mark.parametrize("rows,cols,k", SHAPES)
def test_no_scratch_no_parts(rows, cols, k):
    assert rule(rows, cols, k, None, 0)[0] == 1
    assert rule(rows, cols, k, (1 << 20) + 4, 16)[0] == 1
