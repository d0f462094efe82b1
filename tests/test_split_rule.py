"""The rule that cuts K into parts, on the CPU: where the partial sums go in a scratch at any address, and that the scratch of a plan
serves every smaller batch as well."""
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


# (planned batch, rows an image, columns, terms): heads, 3x3 and 1x1 layers of the small planes, a GEMM whose rows are any number
PLANS = [(128, 1, 1000, 2048), (256, 1, 1000, 2048), (128, 1, 4096, 9216), (32, 49, 512, 4608), (64, 196, 256, 2304), (256, 49, 2048, 512),
         (1500, 1, 33, 1001), (700, 1, 300, 4096)]


@pytest.mark.parametrize("batch,rows,cols,k", PLANS)
def test_the_planned_scratch_serves_smaller_batches(batch, rows, cols, k):
    """Every batch up to the planned one is cut with the plan's scratch as it would be with any amount of it."""
    base = 1 << 20
    wanted = rule(batch * rows, cols, k, None, 0)[1]
    for b in range(1, batch + 1):
        assert rule(b * rows, cols, k, base, wanted)[0] == rule(b * rows, cols, k, base, 1 << 50)[0], b


@pytest.mark.parametrize("rows,cols,k", SHAPES)
def test_a_short_scratch_takes_fewer_parts(rows, cols, k):
    base = 1 << 20
    best = rule(rows, cols, k, base, 1 << 50)[0]
    one = -(-rows // 128) * 128 * -(-cols // (32 if cols <= 32 else 64 if cols <= 64 else 128)) * (32 if cols <= 32 else 64 if cols <= 64 else 128) * 4
    for fit in range(best + 1):
        got = rule(rows, cols, k, base, fit * one)[0]
        assert got <= max(fit, 1)
        if fit == best:
            assert got == best
    assert rule(rows, cols, k, base, (best - 1) * one)[0] > 1 or best == 2
