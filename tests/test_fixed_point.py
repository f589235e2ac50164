"""Key coordinates in fixed point (csrc/stc_fixed.cuh, compiled for the host
here) against the double arithmetic they stand for, on random CTFs and on
fields next to rounding boundaries: where the fixed point decides, it decides
as the double expression does, and it decides nearly always."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "stcdb_gb300", "csrc")

SHIM = r"""
#define __host__
#define __device__
#define __forceinline__ inline
#include "stc_fixed.cuh"
using namespace stc;
extern "C" void boxes(const float *mbr, float wx, float wy, float le, double mx, double my, double me, size_t n,
                      const unsigned long long *f, float *out, unsigned char *ok) {
  const FixedBox b = fixed_box(mbr, wx, wy, le, mx, my, me);
  for (size_t i = 0; i < n; i++, f += 4, out += 4) {
    long long ux = 0, uy = 0, none;
    ok[i] = fixed_to_float(b.x0 + (long long)(f[0] * b.kx), b.e, b.q, out[0], ux) &&
            fixed_to_float(b.y0 + (long long)(f[1] * b.ky), b.e, b.q, out[1], uy) &&
            fixed_to_float(ux + (long long)(f[2] * b.ke), b.e, b.q, out[2], none) &&
            fixed_to_float(uy + (long long)(f[3] * b.ke), b.e, b.q, out[3], none);
  }
}
extern "C" void cells(double a, double b, double d, double lowmax, double edgemax, size_t n,
                      const unsigned long long *low, const unsigned long long *edge, unsigned *out,
                      unsigned char *ok) {
  const FixedAxis x = fixed_axis(a, b, d, lowmax, edgemax);
  for (size_t i = 0; i < n; i++) {
    bool sure = x.e != ~0ull;
    sure &= fixed_cell(low[i] * x.kl, x.e, out[2 * i]) || low[i] == 0;
    sure &= fixed_cell(low[i] * x.kl + edge[i] * x.ke, x.e, out[2 * i + 1]) || edge[i] == 0;
    ok[i] = sure;
  }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, so = d / "s.cpp", d / "s.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    return ctypes.CDLL(str(so))


def _ctf(rng):
    base = rng.choice([0.0, 1e-3, 1.0, 41.0, -87.0, 179.0, -5e4]) + rng.uniform(-1, 1) * 10 ** rng.uniform(-6, 0)
    lo = np.float32([base, rng.uniform(-90, 90)])
    hi = (lo + np.float32(10 ** rng.uniform(-5, 0.5, 2))).astype(np.float32)
    bits = rng.integers(1, 14, 2).tolist()
    return lo, hi, bits + [max(bits)]


def _box64(lo, w, le, m, f):
    """CTF::new_parse_mbr_f_box: double arithmetic, stored as float."""
    x = (np.float64(lo[0]) + f[:, 0] / m[0] * np.float64(w[0])).astype(np.float32)
    y = (np.float64(lo[1]) + f[:, 1] / m[1] * np.float64(w[1])).astype(np.float32)
    z = (x.astype(np.float64) + f[:, 2] / m[2] * np.float64(le)).astype(np.float32)
    t = (y.astype(np.float64) + f[:, 3] / m[2] * np.float64(le)).astype(np.float32)
    return np.stack([x, y, z, t], 1)


def test_decoded_boxes(lib):
    rng = np.random.default_rng(1)
    decided = total = 0
    for _ in range(300):
        lo, hi, bits = _ctf(rng)
        w = (hi - lo).astype(np.float32)
        le = np.float32(max(w))
        m = [float(2 ** b - 1) for b in bits]
        n = 2000
        f = np.stack([rng.integers(0, 2 ** bits[k], n) for k in (0, 1, 2, 2)], 1).astype(np.uint64)
        f[:4] = [[0] * 4, [2 ** bits[0] - 1, 2 ** bits[1] - 1, 2 ** bits[2] - 1, 0], [1] * 4, [0, 0, 1, 1]]
        want = _box64(lo, w, le, m, f.astype(np.float64))
        out, ok = np.zeros((n, 4), np.float32), np.zeros(n, np.uint8)
        mbr = np.concatenate([lo, hi])
        lib.boxes(mbr.ctypes.data_as(ctypes.c_void_p), ctypes.c_float(w[0]), ctypes.c_float(w[1]), ctypes.c_float(le),
                  ctypes.c_double(m[0]), ctypes.c_double(m[1]), ctypes.c_double(m[2]), ctypes.c_size_t(n),
                  f.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p),
                  ok.ctypes.data_as(ctypes.c_void_p))
        good = ok != 0
        assert out[good].tobytes() == want[good].tobytes()
        if abs(lo[0]) > 0.5 and abs(lo[1]) > 0.5:
            decided += good.sum()
            total += n
    assert decided > 0.99 * total


def test_boxes_that_are_left_to_double(lib):
    """Empty, NaN and infinite CTF boxes, and fields of 24 bits and more."""
    out, ok, f = np.zeros(4, np.float32), np.ones(1, np.uint8), np.ones(4, np.uint64)
    for mbr, m in [([1, 1, 0, 0], 15.0), ([np.nan, 1, 2, 2], 15.0), ([1, 1, np.inf, 2], 15.0), ([1, 1, 2, 2], 2.0**24),
                   ([1, 1, 2, 2], 0.0)]:
        b = np.float32(mbr)
        w = b[2:] - b[:2]
        lib.boxes(b.ctypes.data_as(ctypes.c_void_p), ctypes.c_float(w[0]), ctypes.c_float(w[1]),
                  ctypes.c_float(max(w)), ctypes.c_double(m), ctypes.c_double(m), ctypes.c_double(m),
                  ctypes.c_size_t(1), f.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p),
                  ok.ctypes.data_as(ctypes.c_void_p))
        assert not ok[0]


def test_filed_cells(lib):
    rng = np.random.default_rng(2)
    decided = total = 0
    for _ in range(300):
        lo, hi, bits = _ctf(rng)
        w = (hi - lo).astype(np.float32)
        le, m0 = float(max(w)), float(lo[0])
        if not w[0] > 0:
            continue
        g = int(2 ** rng.integers(4, 9))
        scale = g / (float(hi[0]) - m0)
        lowmax, edgemax = float(2 ** bits[0] - 1), float(2 ** bits[2] - 1)
        a, b = scale * float(w[0]) / lowmax, scale * le / edgemax
        d = scale * (max(abs(float(v)) for v in (*lo, *hi)) + le + 1.0) * 2.0 ** -46
        n = 3000
        low, edge = (rng.integers(0, 2 ** k, n).astype(np.uint64) for k in (bits[0], bits[2]))
        k = rng.integers(0, g + 2, n // 2)  # half of them next to cell edges
        low[: n // 2] = np.clip(np.floor(k / a + rng.integers(-1, 2, n // 2)), 0, lowmax).astype(np.uint64)
        box0 = m0 + low.astype(np.float64) / lowmax * float(w[0])
        box2 = box0 + edge.astype(np.float64) / edgemax * le
        want = np.stack([np.floor((box0 - m0) * scale), np.floor((box2 - m0) * scale)], 1)
        out, ok = np.zeros((n, 2), np.uint32), np.zeros(n, np.uint8)
        lib.cells(ctypes.c_double(a), ctypes.c_double(b), ctypes.c_double(d), ctypes.c_double(lowmax),
                  ctypes.c_double(edgemax), ctypes.c_size_t(n), low.ctypes.data_as(ctypes.c_void_p),
                  edge.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p),
                  ok.ctypes.data_as(ctypes.c_void_p))
        good = ok != 0
        assert np.array_equal(out[good].astype(np.float64), want[good])
        decided += good.sum()
        total += n
    assert decided > 0.9 * total
