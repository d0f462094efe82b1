"""The shared-memory ring of the 1x1 kernel, in a model of its waits on the CPU: two converter groups take the k-blocks in turn and
tell the copies of a ring entry apart by one parity bit.  With every entry met by one group only (an even number of entries) no
order of the copies' arrivals lets a group read an entry before its copy has landed; with an odd number some do."""
import itertools
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dlprimitives_b200", "csrc")


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


def test_the_kernels_take_even_rings():
    """Every depth that the launch code can choose is even."""
    text = open(os.path.join(CSRC, "pointwise_tc.cu")).read()
    rule = re.search(r"r\.s_stages = \(std::min\(MAX_S_STAGES - 1, avail / 2\) \+ 1\) & ~1;", text)
    assert rule and re.search(r"r\.s_stages = q\.has_res \? 2 : 4;", text)
    most = int(re.search(r"MAX_S_STAGES = (\d+)", text).group(1))
    for avail in range(7, 15):
        depth = (min(most - 1, avail // 2) + 1) & ~1
        assert depth % 2 == 0 and 2 <= depth <= most and depth < avail
