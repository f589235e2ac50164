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
#include "stc_rules.cuh"
using namespace stc;
extern "C" unsigned block_jobs_beyond(const unsigned *rows, const unsigned *chunks, unsigned n, unsigned long long room) {
  unsigned sum = 0;  // as the block sums them
  for (unsigned i = 0; i < n; i++) sum += jobs_beyond(rows[i], chunks[i], room);
  return sum;
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
