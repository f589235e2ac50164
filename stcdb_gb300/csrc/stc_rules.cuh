// Rules for sizes that the step's kernels and their host code share, as plain
// functions: the tests compile this header for the host.
#pragma once
#include <cstdint>

namespace stc {

// Jobs beyond one per row block of a leaf's border units (rows row blocks,
// chunks candidate chunks each), for a 32-bit sum over the 256 leaves of a
// block: exact up to `room` (jobs_extra, at most 2^22), one more than that for
// any leaf that has no room anyway. (A crowd's leaf of 40M units and 65k
// members has 5e9 of them: the sum of the exact numbers wrapped, looked as if
// it had room, and the jobs were written behind the list's end.)
__host__ __device__ __forceinline__ uint32_t jobs_beyond(uint32_t rows, uint32_t chunks, unsigned long long room) {
  if (!rows) return 0;
  const unsigned long long n = (unsigned long long)rows * (chunks - 1);
  return (uint32_t)(n <= room ? n : room + 1);
}

}  // namespace stc
