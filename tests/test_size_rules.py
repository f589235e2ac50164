"""The size rules that the step's kernels and host code share
(csrc/stc_rules.cuh, compiled for the host here)."""
import ctypes
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "stcdb_gb300", "csrc")

SHIM = r"""
#define __host__
#define __device__
#define __forceinline__ inline
#include <vector>
#include "stc_rules.cuh"
using namespace stc;
extern "C" unsigned block_jobs_beyond(const unsigned *rows, const unsigned *chunks, unsigned n, unsigned long long room) {
  unsigned sum = 0;  // as the block sums them
  for (unsigned i = 0; i < n; i++) sum += jobs_beyond(rows[i], chunks[i], room);
  return sum;
}
extern "C" void paths(unsigned steps, const unsigned *load, const unsigned *fullest, const unsigned *live, unsigned cap,
                      unsigned nb, unsigned lag, unsigned *told) {
  PathChoice c;
  unsigned row = 0;  // told steps in a row; one in COUNT_EVERY counts its tiles for the next
  std::vector<bool> known;
  for (unsigned i = 0; i < steps + lag; i++) {
    if (i < steps) {
      told[i] = c.general;
      known.push_back(row % COUNT_EVERY == 0);
      row = c.general ? row + 1 : 0;
    }
    if (i < lag) continue;
    const unsigned j = i - lag;  // the state that is taken after step i was issued
    const unsigned long long slots = (unsigned long long)nb * TILE_SLOTS;
    if (told[j]) c.step_done(true, known[j] ? live[j] : LOAD_UNKNOWN, live[j], cap, nb, slots);
    else c.step_done(false, known[j] ? load[j] : LOAD_UNKNOWN, fullest[j], cap, nb, slots);
  }
}
extern "C" unsigned handed_out(const unsigned *stack, unsigned index, unsigned size) {
  return ids_handed_out(stack, index, size);
}
extern "C" unsigned cap_auto(unsigned long long n, unsigned nb) { return bin_cap_auto(n, nb); }
extern "C" unsigned cap_grown(unsigned cap, unsigned long long fullest, unsigned long long hits, unsigned nb) {
  return bin_cap_grown(cap, fullest, hits, nb);
}
extern "C" void shape_of(unsigned job_chunk, unsigned refine_bps, unsigned hits_bps, unsigned *out) {
  out[0] = jobs_may_share(job_chunk);
  out[1] = job_chunk_of(job_chunk);
  out[2] = refine_bps_of(refine_bps);
  out[3] = hits_bps_of(hits_bps);
}
extern "C" void builtin_shape(unsigned *out) {
  out[0] = JOB_CHUNK_BUILTIN;
  out[1] = REFINE_BPS_BUILTIN;
  out[2] = HITS_BPS_BUILTIN;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, so = d / "s.cpp", d / "s.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def test_jobs_beyond_their_room_stay_beyond_it_in_32_bits(lib):
    """The sum over a block's leaves is exact while the list has room for it
    and larger than the room otherwise, however dense the leaves."""
    rng = random.Random(1)
    f = lib.block_jobs_beyond
    f.restype = ctypes.c_uint
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint, ctypes.c_ulonglong]
    wraps = 0
    for trial in range(3000):
        room = rng.choice([1 << 22, (1 << 16) + 16 * rng.randrange(1, 1 << 18)])
        n = rng.choice([1, 2, 7, 256])
        big = rng.choice([8, 200, 1 << 14, 3_000_000])  # row blocks of 32 units
        rows = [rng.choice([0, 1, rng.randrange(1, big)]) for _ in range(n)]
        chunks = [rng.choice([1, 2, 33, rng.randrange(1, 4097)]) if r else 1 for r in rows]
        if trial == 0:
            rows, chunks = [1_398_102], [3073]  # 2^32 + 2048 when multiplied out
        true = sum(r * (c - 1) for r, c in zip(rows, chunks))
        wraps += true > room and true % (1 << 32) <= room
        got = f((ctypes.c_uint * n)(*rows), (ctypes.c_uint * n)(*chunks), len(rows), room)
        assert got == true if true <= room else got > room, (rows, chunks, room)
    assert wraps > 0


def _shape(lib, *given):
    out = (ctypes.c_uint * 4)()
    lib.shape_of(*given, out)
    return tuple(out)


def test_the_built_in_launch_shape_is_the_automatic_one(lib):
    """The autotuner names the built-in values where its first runs, which it
    compares the later ones with, left them at 0: both run the same way."""
    b = (ctypes.c_uint * 3)()
    lib.builtin_shape(b)
    auto = _shape(lib, 0, 0, 0)
    assert _shape(lib, *b) == auto == (1, 8, 0, 16)
    for chunk, bps, hits in [(1, 1, 1), (7, 4, 8), (9, 9, 32), (64, 32, 64)]:
        assert _shape(lib, chunk, bps, hits) == (0, chunk, bps, hits)  # others as given
    assert _shape(lib, 1000, 1000, 1000) == (0, 64, 32, 64)


REC = 32   # bytes of a hit record, and of a table slot
TILE = 768


def _caps(lib):
    u, ll = ctypes.c_uint, ctypes.c_ulonglong
    lib.cap_auto.restype = lib.cap_grown.restype = u
    lib.cap_auto.argtypes = [ll, u]
    lib.cap_grown.argtypes = [u, ll, ll, u]
    return lib.cap_auto, lib.cap_grown


def test_automatic_hit_bins_follow_the_objects_and_stay_small_beside_the_table(lib):
    auto, _ = _caps(lib)
    for log2 in (10, 16, 20, 24, 28, 30, 32, 33):
        slots = 1 << log2
        nb = (slots + TILE - 1) // TILE
        for n in (1, 1000, 100_003, 300_000, 1_000_000, 10_000_000, 100_000_000):
            cap = auto(n, nb)
            room = max(1 << 22, 8 * n)
            assert cap % 16 == 0 and cap >= 16
            assert nb * cap >= room or cap == 1 << 24
            # a quarter and two standard deviations more, 8 more and whole chunks a bin
            assert nb * cap <= 1.25 * (room + nb) + 2 * (nb * (room + nb)) ** 0.5 + 24 * nb
    # 300k objects in 2^28 slots had 0.89 GB of bins, 1M in 2^30 3.6 GB
    assert auto(300_000, (1 << 28) // TILE + 1) * ((1 << 28) / TILE) * REC < 0.4e9
    assert auto(1_000_000, (1 << 30) // TILE + 1) * ((1 << 30) / TILE) * REC < 1.5e9


def test_hit_bins_grow_with_the_hits_not_with_one_crowd(lib):
    _, grown = _caps(lib)
    nb = (1 << 28) // TILE + 1
    assert grown(80, 80, 10 ** 6, nb) == 80                     # nothing to grow for
    assert grown(32, 781, 1_500_000, nb) == 48                  # one crowd of 1600 objects: 0.5 GB, not 10.9
    assert grown(64, 781, 1_500_000, nb) == 64                  # never less
    assert grown(64, 100, 35_000_000, nb) == 144  # an even crowd gets what it asks
    assert grown(64, 5000, 350_000_000, nb) == 704              # what the tiled path can use
    rng = random.Random(3)
    for _ in range(2000):
        nb = rng.randrange(1, 1 << 22)
        cap = 16 * rng.randrange(1, 60)
        hits = rng.randrange(1, 1 << rng.randrange(4, 36))
        fullest = rng.randrange(1, max(hits, 2))
        got = grown(cap, fullest, hits, nb)
        assert cap <= got <= max(cap, 704)
        assert got == cap or got * nb <= max(8 * hits + 8 * nb, 48 * nb)
        if fullest > cap and fullest * 1.25 + 32 <= min(704, 8 * hits / nb):
            assert got >= fullest * 1.25


def test_ids_handed_out_are_found_from_the_free_stack(lib):
    """Splits take four ids off the stack, merges put four back; the bound the
    context itself keeps (the deepest the stack was ever taken to) is found
    again from the stack, or a lower one that still covers every id in use
    and every id that the stack hands out before its untouched end."""
    f = lib.handed_out
    f.restype = ctypes.c_uint
    f.argtypes = [ctypes.c_void_p, ctypes.c_uint, ctypes.c_uint]
    rng = random.Random(11)
    for _ in range(200):
        size = rng.choice([64, 400, 4000])
        stack, index, used, deepest = list(range(size)), 1, [0], 1
        groups = []
        for _ in range(rng.randrange(0, 200)):
            if index + 4 <= size and (not groups or rng.random() < 0.55):
                groups.append(stack[index:index + 4])
                index += 4
                deepest = max(deepest, index)
            elif groups:
                for i in groups.pop(rng.randrange(len(groups))):
                    index -= 1
                    stack[index] = i
        used = [0] + [i for g in groups for i in g]
        high = f((ctypes.c_uint * size)(*stack), index, size)
        assert index <= high <= deepest
        assert max(used) < max(high, 1)
        assert all(i < high for i in stack[index:high])
        assert stack[high:] == list(range(high, size))
    assert f((ctypes.c_uint * 8)(*range(8)), 8, 8) == 8 and f((ctypes.c_uint * 8)(*range(8)), 3, 8) == 3


def _told(lib, load, fullest, live, cap=704, nb=1000, lag=0):
    n = len(load)
    arr = [(ctypes.c_uint * n)(*v) for v in (load, fullest, live)]
    out = (ctypes.c_uint * n)()
    lib.paths(n, *arr, cap, nb, lag, out)
    return list(out)


@pytest.mark.parametrize("lag", [0, 1, 2])
def test_steps_are_told_to_be_general_while_the_tiles_would_not_do(lib, lag):
    n = 600
    fits, full = ([300] * n, [150] * n, [150] * n), ([800] * n, [400] * n, [400] * n)
    assert _told(lib, *fits, lag=lag) == [0] * n
    for cap, nb in [(704, 1000), (40, 1000)]:  # too full tiles, or bins that may not grow
        assert _told(lib, *full, cap=cap, nb=nb, lag=lag) == [0] * (1 + lag) + [1] * (n - 1 - lag)
    assert sum(_told(lib, *fits, cap=140, lag=lag)) > 0.8 * n  # tried again, 141 of 140 guessed
    assert _told(lib, *full, nb=13, lag=lag) == [0] * n        # no tiles to choose
    assert _told(lib, *full, nb=4194304, lag=lag)[-1] == 1     # 3 * 2^30 slots
    assert _told(lib, *full, nb=4194305, lag=lag) == [0] * n


@pytest.mark.parametrize("lag", [0, 1, 2])
def test_told_steps_go_back_to_tiles_when_they_would_do(lib, lag):
    """A table that fills up and empties again, and a guess that keeps failing."""
    live = [200] * 50 + [400] * 100 + [340] * 400
    told = _told(lib, [2 * v for v in live], live, live, lag=lag)
    assert sum(told[:50]) == 0 and sum(told[50:150]) >= 99 - lag and sum(told[165:]) == 0
    # few meetings a tile, more hits than fit: tried again ever more seldom
    n = 3000
    told = _told(lib, [800] * n, [10] * n, [100] * n, lag=lag)
    assert sum(told[:100]) > 50 and sum(told[500:]) > 0.9 * (n - 500)
