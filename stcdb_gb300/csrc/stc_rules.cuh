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

// Launch shape of the refinement (stc_config.job_chunk, refine_blocks_per_sm).
// The built-in value, given or not, leaves the choice to the library: jobs
// taken by demand where that is faster (job_shares), more blocks where the
// last warps are a larger part of the time (refine_blocks). So the autotuner's
// settings, which name every field, hold what its runs with the fields left at
// 0 were timed with.
constexpr uint32_t JOB_CHUNK_BUILTIN = 8, REFINE_BPS_BUILTIN = 8, HITS_BPS_BUILTIN = 16;
constexpr uint32_t JOB_CHUNK_MOST = 64, REFINE_BPS_MOST = 32, HITS_BPS_MOST = 64;
inline bool jobs_may_share(uint32_t job_chunk) { return job_chunk == 0 || job_chunk == JOB_CHUNK_BUILTIN; }
inline uint32_t job_chunk_of(uint32_t given) {
  return given == 0 ? JOB_CHUNK_BUILTIN : given < JOB_CHUNK_MOST ? given : JOB_CHUNK_MOST;
}
// Blocks an SM of the pair tests, 0: the library's choice.
inline uint32_t refine_bps_of(uint32_t given) {
  return given == REFINE_BPS_BUILTIN ? 0 : given < REFINE_BPS_MOST ? given : REFINE_BPS_MOST;
}
inline uint32_t hits_bps_of(uint32_t given) {
  return given == 0 ? HITS_BPS_BUILTIN : given < HITS_BPS_MOST ? given : HITS_BPS_MOST;
}

}  // namespace stc
