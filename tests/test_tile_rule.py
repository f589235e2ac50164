"""The rule that lets a step take the tiled table update (csrc/stc_table.cu):
runs of tiles worked through one by one, entered with what a few halo tiles
before them carry over, place every key where inserting them one by one in
priority order over the whole ring does."""
import random

import pytest


def insert_all(table, keys, size):
    """Keys (home, priority, id) into the ring in priority order: the first
    empty slot, or the key's own old entry. Returns {id: slot}."""
    taken, placed = dict(table), {}
    for home, _, key in sorted(keys, key=lambda k: k[1]):
        pos = home
        for _ in range(size):
            if taken.get(pos) == key or pos not in taken:
                break
            pos = (pos + 1) % size
        else:
            raise AssertionError("ring full")
        taken[pos] = key
        placed[key] = pos
    return placed


def run_tiles(table, start, tiles, bins, carried):
    """Tiles in ring order with `carried` entering the first; deferred
    acceptance inside each tile. Returns ({id: slot}, keys carried out)."""
    placed = {}
    for j in tiles:
        lo, hi = start[j], start[j + 1]
        walkers = [(max(h, lo) if fresh else lo, pr, key) for fresh, (h, pr, key) in
                   [(False, k) for k in carried] + [(True, k) for k in bins[j]]]
        info = {k[2]: k for k in list(carried) + list(bins[j])}
        random.shuffle(walkers)
        claim, carried = {}, []
        while walkers:
            pos, pr, key = walkers.pop()
            while True:
                if pos == hi:
                    carried.append(info[key])
                    break
                if table.get(pos) == key:
                    placed[key] = pos
                    break
                if pos not in table:
                    if pos not in claim:
                        claim[pos] = (pr, key)
                        break
                    if pr < claim[pos][0]:
                        (pr, key), claim[pos] = claim[pos], (pr, key)
                pos += 1
        for pos, (_, key) in claim.items():
            placed[key] = pos
    return placed, carried


def halo_of(load, tile, limit, most=7):
    """fuse_halo of csrc/stc_insert.cuh."""
    if load >= limit:
        return 0
    for h in range(1, most + 1):
        if load * (h + 1) < tile * h:
            return h
    return 0


@pytest.mark.parametrize("size,tiles,live,new,clump", [(640, 16, 0.25, 0.2, 0), (641, 20, 0.3, 0.25, 0),
                                                       (900, 18, 0.2, 0.1, 12), (1000, 25, 0.1, 0.1, 20),
                                                       (777, 15, 0.45, 0.3, 0)])
def test_tiles_with_a_halo_place_keys_like_sequential_insertion(size, tiles, live, new, clump):
    rng = random.Random(size * 1000 + tiles)
    random.seed(5)
    start = [j * size // tiles for j in range(tiles + 1)]
    smallest = size // tiles
    used = 0
    for _ in range(60):
        table = {s: ("old", s) for s in range(size) if rng.random() < live}
        keys = []
        for i in range(int(new * size)):
            home = rng.randrange(clump) * (size // clump) if clump and rng.random() < 0.3 else rng.randrange(size)
            key = ("new", i)
            if rng.random() < 0.2:  # an old entry of its own a little further on
                pos = (home + rng.randrange(1, 6)) % size
                if table.get(pos, ("old",))[0] == "old":
                    table[pos] = key
            keys.append((home, rng.random(), key))
        bins = [[k for k in keys if start[j] <= k[0] < start[j + 1]] for j in range(tiles)]
        load = max(len(bins[j]) + sum(start[j] <= s < start[j + 1] for s in table) for j in range(tiles))
        halo = halo_of(load, smallest, 0.75 * (size + tiles - 1) // tiles)
        if not halo:
            continue
        used += 1
        want = insert_all(table, keys, size)
        runs = rng.randrange(1, tiles + 1)
        got = {}
        for r in range(runs):
            first, last = r * tiles // runs, (r + 1) * tiles // runs
            before = [(first - halo + q) % tiles for q in range(halo)]
            _, carried = run_tiles(table, start, before, bins, [])
            # carried keys enter at the run's first slot (the ring's slot 0 for run 0)
            placed, _ = run_tiles(table, start, range(first, last), bins, carried)
            got.update({k: p for k, p in placed.items()})
        assert got == want
    assert used > 0 or live > 0.4


def test_rule_bounds():
    assert halo_of(0, 768, 576) == 1
    assert halo_of(383, 768, 576) == 1 and halo_of(384, 768, 576) == 2
    assert halo_of(575, 768, 576) == 3 and halo_of(576, 768, 576) == 0
