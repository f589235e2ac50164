// Packed key coordinates in 64-bit fixed point.
//
// A key's box is stored as integer fields of its CTF's box, and decoded (or
// filed in a cell) by double arithmetic: base + (field / fieldmax) * width.
// Double arithmetic runs at 2 lanes a clock and SM here: a warp's add costs 16
// cycles, a division some 25 of them. The results that are kept are coarser, a
// float or a cell number, so the value is computed as field * k in integer
// units of 2^-q, off by a known number of units, and the double arithmetic is
// left to values so near a rounding boundary that the two could differ.
#pragma once
#include <cmath>
#include <cstdint>
#include <limits>

namespace stc {

// The float nearest to t * 2^-q, and that float in units; false when a value
// within e units of t (or of the float's rounding boundaries) could round to
// another, or is small or out of range.
__host__ __device__ __forceinline__ bool fixed_to_float(long long t, unsigned long long e, int q, float &f,
                                                        long long &units) {
  const unsigned long long a = t < 0 ? 0ull - (unsigned long long)t : (unsigned long long)t;
  if (a < (1ull << 26)) return false;
#ifdef __CUDA_ARCH__
  const int h = 63 - __clzll((long long)a);
#else
  const int h = 63 - __builtin_clzll(a);
#endif
  const int sh = h - 23;
  const unsigned long long half = 1ull << (sh - 1), rem = a & (2 * half - 1);
  if (e >= half / 2 || (rem + e >= half && rem <= half + e)) return false;
  const unsigned long long m = (a >> sh) + (rem > half ? 1ull : 0ull);  // 2^23 to 2^24
  const uint32_t bits = ((uint32_t)(h - q + 127) << 23) + ((uint32_t)m - (1u << 23)) + (t < 0 ? 0x80000000u : 0u);
#ifdef __CUDA_ARCH__
  f = __uint_as_float(bits);
#else
  __builtin_memcpy(&f, &bits, 4);
#endif
  const long long r = (long long)(m << sh);
  units = t < 0 ? -r : r;
  return true;
}

// Decode of a CTF's box fields to floats (CTF::new_parse_mbr_f_box): units
// 2^-q, low corner, units per field unit, error bound. e is ~0 where a CTF
// has to be decoded in double.
struct FixedBox {
  long long x0, y0;
  unsigned long long kx, ky, ke, e;
  int q, pad;
};

inline FixedBox fixed_box(const float mbr[4], float wx, float wy, float le, double mx, double my, double me) {
  FixedBox b{};
  b.e = ~0ull;
  double v = 1.0;
  for (int i = 0; i < 4; i++) v = std::fmax(v, std::fabs((double)mbr[i]));
  const bool sizes = wx >= 0 && wy >= 0 && le >= 0 && mx > 0 && my > 0 && me > 0;
  // fields below 2^24 keep k's rounding (half a unit each) within 2^24 units
  if (!std::isfinite(v) || !std::isfinite((double)le) || !sizes || mx >= 16777216.0 || my >= 16777216.0 ||
      me >= 16777216.0)
    return b;
  v += 2.0 * ((double)wx + (double)wy + (double)le) + 1.0;
  int up = 0;
  std::frexp(v, &up);  // v < 2^up
  if (up > 60) return b;
  b.q = 60 - up;
  b.x0 = std::llrint(std::ldexp((double)mbr[0], b.q));
  b.y0 = std::llrint(std::ldexp((double)mbr[1], b.q));
  b.kx = (unsigned long long)std::llrint(std::ldexp((double)wx / mx, b.q));
  b.ky = (unsigned long long)std::llrint(std::ldexp((double)wy / my, b.q));
  b.ke = (unsigned long long)std::llrint(std::ldexp((double)le / me, b.q));
  // k: half a unit a field unit, and 2^-52 of the product from its own
  // division; the double decode: three roundings of 2^-53 of at most 2^60
  // units; x0, y0: half a unit. Taken four times.
  b.e = 4 * ((unsigned long long)std::fmax(mx, std::fmax(my, me)) + 256 + 3 * 128 + 1);
  return b;
}

// Filing of a CTF's keys on one axis of its cell index: 2^-FIXED_CELL_BITS
// cells per unit of the low and the edge field, error bound; e is ~0 where
// keys have to be filed in double.
constexpr int FIXED_CELL_BITS = 36;
struct FixedAxis {
  unsigned long long kl, ke, e, pad;
};

// a, b: cells per field unit; d: bound on the error of the double filing, in
// cells.
inline FixedAxis fixed_axis(double a, double b, double d, double lowmax, double edgemax) {
  FixedAxis x{0, 0, ~0ull, 0};
  const double top = a * lowmax + b * edgemax;
  if (!(top < 33554432.0) || !(d < 0.25) || !(lowmax < 16777216.0) || !(edgemax < 16777216.0)) return x;
  x.kl = (unsigned long long)std::llrint(std::ldexp(a, FIXED_CELL_BITS));
  x.ke = (unsigned long long)std::llrint(std::ldexp(b, FIXED_CELL_BITS));
  // k: half a unit a field unit, and 2^-50 of the product; d
  x.e = (unsigned long long)(lowmax + edgemax + std::ldexp(top, FIXED_CELL_BITS - 50) +
                             std::ldexp(d, FIXED_CELL_BITS)) + 4;
  return x;
}

// The cell that position t (units) lies in; false when one within e units
// could lie in another.
__host__ __device__ __forceinline__ bool fixed_cell(unsigned long long t, unsigned long long e, uint32_t &cell) {
  cell = (uint32_t)(t >> FIXED_CELL_BITS);
  const unsigned long long frac = t & ((1ull << FIXED_CELL_BITS) - 1);
  return frac >= e && frac + e < (1ull << FIXED_CELL_BITS);
}

}  // namespace stc
