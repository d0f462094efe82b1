"""The shared-memory rings of the 1x1 kernel, in a model of their waits on the CPU, at the depths that its launches choose.

The A ring: two converter groups take the k-blocks in turn and tell the copies of a ring entry apart by one parity bit.  With every
entry met by one group only (an even number of entries) no order of the copies' arrivals lets a group read an entry before its
copy has landed; with an odd number some do.

The epilogue buffers of a launch with a residual: two sets of epilogue warps take the groups of 32 channels in turn and wait for the
residual operand of their group in the same way."""
import ctypes
import itertools

import pytest


def rings(bn, kblocks, resident, residual):
    from dlprimitives_b200 import capi
    a, e = ctypes.c_int(), ctypes.c_int()
    capi.check(capi.lib().dlp_pointwise_rings(bn, kblocks, resident, residual, ctypes.byref(a), ctypes.byref(e)))
    return a.value, e.value


# every launch there is: column tile, k-blocks, weights resident (at most 128 KB: 2 * bn * 32 floats a k-block) or streaming, residual
LAUNCHES = [(bn, kb, res_w, residual) for bn in (32, 64, 128) for kb in range(1, 9) for res_w in (0, 1) for residual in (0, 1)
            if not res_w or kb * 2 * bn * 32 * 4 <= 128 * 1024]


def reads_too_early(entries, order):
    """Copies 0 .. entries-1 land in the given order; after each landing both groups go as far as their waits let them (nothing
    else holds them up before the tensor-memory ring is full: two k-blocks each).  True if a group read a copy that had not landed."""
    phase, landed, at = [0] * entries, set(), [0, 1]
    for copy in order:
        landed.add(copy)
        phase[copy % entries] += 1
        moved = True
        while moved:
            moved = False
            for g in (0, 1):
                it = at[g]
                if it >= g + 4 or (phase[it % entries] & 1) == ((it // entries) & 1):       # ring full, or the parity wait holds
                    continue
                if it not in landed:
                    return True
                at[g] += 2
                moved = True
    return False


@pytest.mark.parametrize("entries", [2, 4, 6])
def test_even_rings_are_never_read_early(entries):
    assert not any(reads_too_early(entries, order) for order in itertools.permutations(range(entries)))


def test_odd_rings_can_be():
    assert any(reads_too_early(3, order) for order in itertools.permutations(range(3)))


def residual_read_early(buffers, groups, tiles=8, handback=True):
    """Every interleaving of: the copy thread arming the next group's buffer, a copy landing (in any order), and each of two
    sets taking its next group -- the accumulator of its tile, which is there once both sets have read the one two tiles back, then the
    parity wait, the hand-back of the accumulator after its last group, and the hand-back of the buffer.  True if some order
    lets a set read a residual that has not landed.  handback=False: accumulators hold nobody up (buffers have to be safe by themselves)."""
    total = groups * tiles
    seq = [list(range(s, total, 2)) for s in (0, 1)]           # the groups of each set, in order

    def full(state, j):                                        # the parity wait for copy j
        armed, flying, done = state[0], state[1], state[2]
        landed = sum(1 for c in range(j % buffers, armed, buffers) if c not in flying)
        return (landed & 1) != ((j // buffers) & 1)

    start = (0, frozenset(), (0, 0), (0, 0))                   # copies armed, copies in flight, groups read, groups handed back per set
    seen, stack = {start}, [start]
    while stack:
        armed, flying, read, back = stack.pop()
        nxt = []
        if armed < total:
            # waits until the buffer's last group is handed back, by parity as well
            handed = sum(1 for s in (0, 1) for c in seq[s][:back[s]] if c % buffers == armed % buffers)
            if (handed & 1) == ((armed // buffers) & 1):
                nxt.append((armed + 1, flying | {armed}, read, back))
        for c in flying:
            nxt.append((armed, flying - {c}, read, back))
        for s in (0, 1):
            if read[s] > back[s]:
                nxt.append((armed, flying, read, tuple(b + (i == s) for i, b in enumerate(back))))
            elif read[s] < len(seq[s]):
                j = seq[s][read[s]]
                per_tile = groups // 2
                free = not handback or min(read) >= (j // groups - 1) * per_tile
                if free and full((armed, flying, None), j):
                    if j >= armed or j in flying:
                        return True
                    nxt.append((armed, flying, tuple(r + (i == s) for i, r in enumerate(read)), back))
        for st in nxt:
            if st not in seen:
                seen.add(st)
                stack.append(st)
    return False


def test_three_epilogue_buffers_are_read_early():
    assert residual_read_early(3, 2)


@pytest.mark.parametrize("buffers", [2, 4, 6])
@pytest.mark.parametrize("groups", [2, 4])
def test_even_epilogue_buffers_never_are(buffers, groups):
    assert not residual_read_early(buffers, groups, tiles=6, handback=False)


@pytest.mark.parametrize("launch", LAUNCHES)
def test_the_launches_take_even_rings(launch):
    """An even number of A slots, and with a residual and two sets of epilogue warps (tiles of 64 channels and more) of buffers; no
    more than fit beside the weights."""
    bn, kblocks, resident, residual = launch
    slots, buffers = rings(*launch)
    assert slots in (2, 4, 6)
    assert buffers >= 2
    if residual and bn > 32:
        assert buffers % 2 == 0
    weights = (kblocks if resident else 4) * 2 * bn * 32 * 4
    assert 2048 + weights + (slots + buffers) * 16384 <= 227 * 1024
