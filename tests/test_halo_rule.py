"""The shipped rule of the tiled table update's halo (halo_tiles of
csrc/stc_rules.cuh, compiled for the host here), over all halos it gives: at
the fullest tiles it accepts, runs entered with what the halo carries place
every key where inserting them one by one does."""
import ctypes
import os
import random
import subprocess

import pytest

from test_tile_rule import insert_all, run_tiles

CSRC = os.path.join(os.path.dirname(__file__), "..", "stcdb_gb300", "csrc")

SHIM = r"""
#define __host__
#define __device__
#define __forceinline__ inline
#include "stc_rules.cuh"
using namespace stc;
extern "C" unsigned halo(unsigned long long load, unsigned nb, unsigned long long slots) {
  return halo_tiles(load, nb, slots);
}
extern "C" void limits(unsigned *out) {
  out[0] = MAX_HALO;
  out[1] = MIN_TILES;
  out[2] = TILE_LOAD;
  out[3] = TILE_SLOTS;
}
"""


@pytest.fixture(scope="module")
def halo(tmp_path_factory):
    d = tmp_path_factory.mktemp("halo")
    src, so = d / "s.cpp", d / "s.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    out = (ctypes.c_uint * 4)()
    lib.limits(out)
    lib.halo.restype = ctypes.c_uint
    lib.halo.argtypes = [ctypes.c_ulonglong, ctypes.c_uint, ctypes.c_ulonglong]
    return lib.halo, tuple(out)


def test_the_rule_at_its_limits(halo):
    f, (most, fewest, load, slots) = halo
    assert (most, fewest, load, slots) == (15, 14, 704, 768)
    nb = 1 << 20
    assert f(0, nb, slots) == 1 and f(383, nb, slots) == 1 and f(384, nb, slots) == 2
    assert f(576, nb, slots) == 4 and f(703, nb, slots) == 11 and f(704, nb, slots) == 0
    assert f(0, 13, slots) == 0 and f(0, 14, slots) == 1  # too small a table
    assert f(600, 14, slots) == 4 and f(680, 14, slots) == 0  # at most half of the tiles: 8 of 14 is too many
    for c in range(load):
        h = f(c, nb, slots)
        assert h and c * (h + 1) < slots * h and (h == 1 or c * h >= slots * (h - 1))
    # smaller tiles (the table's last slots decide their size): up to 15 halo tiles
    assert f(99, nb, 106) == 15 and f(100, nb, 106) == 0


@pytest.mark.parametrize("h", range(1, 16))
@pytest.mark.parametrize("clumped", [False, True])
def test_runs_behind_the_longest_halo_of_a_load_place_keys_like_sequential_insertion(halo, h, clumped):
    """Tiles filled to the most that halo h is given for: occupied slots and
    new keys, in the clumped case homed in the tile's last slots, so that as
    many as possible are carried on."""
    f, _ = halo
    tiles = 2 * h + 6 if h > 4 else 14
    slots = max(h, 4) * (h + 1)
    size = tiles * slots
    c = max(h, 4) * h - 1  # the most with c * (h + 1) < slots * h; too much for a halo of h - 1
    assert f(c, tiles, slots) == h
    rng = random.Random(100 * h + clumped)
    random.seed(h)
    carried_most = 0
    for _ in range(max(2, 24 // h)):
        start = [j * slots for j in range(tiles + 1)]
        table, keys = {}, []
        for j in range(tiles):
            live = rng.randrange(c + 1)
            for s in rng.sample(range(start[j], start[j + 1]), live):
                table[s] = ("old", s)
            for i in range(c - live if rng.random() < 0.7 else rng.randrange(c - live + 1)):
                home = start[j + 1] - 1 - rng.randrange(3) if clumped else rng.randrange(start[j], start[j + 1])
                keys.append((home, rng.random(), ("new", j, i)))
        bins = [[k for k in keys if start[j] <= k[0] < start[j + 1]] for j in range(tiles)]
        assert max(len(bins[j]) + sum(start[j] <= s < start[j + 1] for s in table) for j in range(tiles)) <= c
        want = insert_all(table, keys, size)
        runs = rng.randrange(1, tiles + 1)
        got = {}
        for r in range(runs):
            first, last = r * tiles // runs, (r + 1) * tiles // runs
            _, carried = run_tiles(table, start, [(first - h + q) % tiles for q in range(h)], bins, [])
            carried_most = max(carried_most, len(carried))
            placed, _ = run_tiles(table, start, range(first, last), bins, carried)
            got.update(placed)
        assert got == want
    assert carried_most > 0 or not clumped
