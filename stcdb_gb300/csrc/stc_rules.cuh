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

// Ids that a free stack of `size` entries (entry i holds id i until it is taken;
// the entries below `index` are taken) ever handed out lie below this: behind
// the last entry that holds another id than its own, everything is as it was.
inline uint32_t ids_handed_out(const uint32_t *stack, uint32_t index, uint32_t size) {
  uint32_t high = size;
  while (high > index && stack[high - 1] == high - 1) high--;
  return high;
}

// Tiles of the meeting table (stc_table.cu) and the bins of a step's hits.
constexpr uint32_t TILE_SLOTS = 768;    // largest tile
constexpr uint32_t TILE_LOAD = 704;     // (occupied slots + hits) of a tile stay below this on the tiled path
constexpr uint32_t HIT_CHUNK = 16;      // records of a bin that lie together (hit_place)

// Halo tiles the tiled table update needs for a step whose fullest tile has
// `load` occupied slots and hits, in a table of nb tiles of `slots` slots or
// one more; 0: the step takes the general path (k_hits, k_insert_ordered,
// k_sweep). Why that many, see stc_table.cu.
constexpr uint32_t MAX_HALO = 15;
constexpr uint32_t MIN_TILES = 14;  // a smaller table is not worth tiles
__host__ __device__ __forceinline__ uint32_t halo_tiles(unsigned long long load, uint32_t nb,
                                                        unsigned long long slots) {
  if (nb < MIN_TILES || load >= TILE_LOAD) return 0;  // the carry lists hold TILE_LOAD hits
  for (uint32_t h = 1; h <= MAX_HALO && 2 * h <= nb; h++)
    if (load * (h + 1) < slots * h) return h;
  return 0;
}

// What general steps do, and whether the next step is told beforehand to be one,
// from each step's counters. A step that the tiles cannot take finds its hits in
// bins and updates the table bin by bin (k_hits). A step told to be general
// leaves them in sequence, and its table update runs beside the pair tests
// (k_hits_part), which also spreads a crowded table's long walks: general steps
// of the stress model by bins and told, ms, at 0.35 to 0.59 meetings a slot: 200k
// objects (1.3 to 2.1 GB of slots) 4.4 and 3.9, 5.2 and 5.0, 34 and 18; 700k (19
// GB) 55 and 47; 1M (34 GB) 107 and 88; 1.4M (69 GB) 165 and 134. A larger table
// is out of reach of the address translation, and the bins' locality counts for
// more: at 137 GB 1.9M objects 274 and 390, the hotspot model at 10M 340 and 460.
// So a step that the tiles could not take tells the next ones, in tables of up
// to TOLD_MOST_SLOTS (103 GB).
// Told steps cannot see whether the tiles would do again. The fullest tile of
// the step before is the guess: its meetings, and a hit for each, less a
// sixteenth, since the tile with most meetings is seldom the one with most
// hits. It can be wrong (hits of one tile whose meetings lie in the next): a
// wrong one is followed by twice as many told steps as the last, up to 64.
// Told steps count their tiles' meetings one time in COUNT_EVERY: the marks
// cost the sweep of 507M meetings 4.7 of 14.4 ms.
constexpr uint64_t TOLD_MOST_SLOTS = 3ull << 30;
constexpr uint64_t LOAD_UNKNOWN = ~0ull;  // the step before did not count
constexpr uint32_t COUNT_EVERY = 8;
struct PathChoice {
  bool general = false;  // tell the next step
  uint32_t wait = 0, next_wait = 2;
  // One step, in the order of their issue. told: it was told to. load: meetings
  // and hits of its fullest tile (told: meetings of the step before). fullest:
  // hits of its fullest bin (told: not used). cap: records a bin may have.
  // slots: of the table.
  void step_done(bool told, uint64_t load, uint64_t fullest, uint32_t cap, uint32_t nb, uint64_t slots) {
    if (nb < MIN_TILES || slots > TOLD_MOST_SLOTS) return;
    if (told) {
      if (wait) wait--;
      if (wait || load == LOAD_UNKNOWN) return;
      const uint64_t guess = load - load / 16;
      if (guess <= cap && halo_tiles(2 * guess, nb, slots / nb)) general = false;
      return;
    }
    if (load == LOAD_UNKNOWN) return;  // a told one before it did not count; the next one shows
    general = fullest > cap || !halo_tiles(load, nb, slots / nb);
    if (!general) {
      next_wait = 2;
      return;
    }
    wait = next_wait;
    next_wait = next_wait < 64 ? 2 * next_wait : 64;
  }
};

// Records per bin when `total` are spread over nb bins, rounded up (at least 1;
// a run of bins stays below 2^32 records).
inline uint32_t bin_share(uint64_t total, uint32_t nb) {
  const uint64_t n = (total + nb - 1) / nb;
  return (uint32_t)(n < 1 ? 1 : n > (1u << 24) ? 1u << 24 : n);
}

// Records per bin of an automatic hit buffer (stc_config.hit_capacity 0) for n
// objects: room for 4M or 8 n hits, a quarter and two standard deviations of
// an even spread more, in whole chunks. A table of many slots for few objects
// has 16 records a tile, 2% of its slots' memory. (With 64 more a bin whatever
// its share, 2^30 slots took 2.9 GB and 2^32 slots 11.5.)
inline uint32_t bin_cap_auto(uint64_t n, uint32_t nb) {
  const uint64_t share = bin_share(8 * n > (1u << 22) ? 8 * n : 1u << 22, nb);
  uint64_t root = 0;
  while ((root + 1) * (root + 1) <= share) root++;
  const uint64_t cap = (share + share / 4 + 2 * root + 8 + HIT_CHUNK - 1) / HIT_CHUNK * HIT_CHUNK;
  return (uint32_t)(cap > (1u << 24) ? 1u << 24 : cap);
}

// Records per bin after a step of `hits` hits whose fullest bin had `fullest`:
// a quarter more than that, but no more than eight times the mean bin (or 48
// records, a sixteenth of the slots' memory) and no more than the tiled path
// can use. One crowd's bin must not size all the others: 1600 objects of
// neighbouring ids fill one tile, and 2^28 slots then took 10.9 GB for it.
inline uint32_t bin_cap_grown(uint32_t cap, uint64_t fullest, uint64_t hits, uint32_t nb) {
  if (fullest <= cap) return cap;
  uint64_t most = 8 * (uint64_t)bin_share(hits, nb);
  if (most < 48) most = 48;
  if (most > TILE_LOAD) most = TILE_LOAD;
  uint64_t want = (fullest + fullest / 4 + 2 * HIT_CHUNK - 1) / HIT_CHUNK * HIT_CHUNK;
  if (want > most) want = most / HIT_CHUNK * HIT_CHUNK;
  return want > cap ? (uint32_t)want : cap;
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
