"""The object queries' search (csrc/stc_query.cu, first_of), five levels of the
reference's binary search a round, against that search one step at a time:
the same answer and the same positions looked at, on sorted and on any data."""
import random

import pytest


def one_by_one(keys, pid):
    low, high, find, seen = 0, len(keys) - 1, -1, []
    while low <= high:
        mid = low + (high - low) // 2
        seen.append(mid)
        if keys[mid] == pid:
            find = mid
        if keys[mid] >= pid:
            high = mid - 1
        else:
            low = mid + 1
    return find, seen


def by_rounds(keys, pid):
    low, high, find, seen = 0, len(keys) - 1, -1, []

    def bounds(h):
        lo, hi = low, high
        for b in range(h.bit_length() - 2, -1, -1):
            if lo > hi:
                break
            mid = lo + (hi - lo) // 2
            if (h >> b) & 1:
                lo = mid + 1
            else:
                hi = mid - 1
        return lo, hi

    while low <= high:
        at = {}
        for lane in range(1, 32):
            lo, hi = bounds(lane)
            if lo <= hi:
                at[lane] = lo + (hi - lo) // 2
                assert 0 <= at[lane] < len(keys)
        h, last = 1, 0
        while h < 32 and h in at:
            seen.append(at[h])
            if keys[at[h]] == pid:
                last = h
            h = 2 * h + (keys[at[h]] < pid)
        if last:
            find = at[last]
        low, high = bounds(h)
    return find, seen


@pytest.mark.parametrize("n", [0, 1, 2, 3, 30, 31, 32, 33, 62, 63, 64, 1000, 1023, 1024, 1025])
def test_rounds_search_as_one_by_one(n):
    rng = random.Random(n)
    for spread in (1, 3, n + 2, 8 * n + 8):
        keys = sorted(rng.randrange(spread) for _ in range(n))
        mixed = keys[:]
        rng.shuffle(mixed)
        for pid in {0, spread // 2, spread - 1, spread, *(rng.choice(keys) for _ in range(min(n, 8)))}:
            assert by_rounds(keys, pid) == one_by_one(keys, pid)
            assert by_rounds(mixed, pid) == one_by_one(mixed, pid)
        if keys:
            pid = rng.choice(keys)
            assert by_rounds(keys, pid)[0] == keys.index(pid)
