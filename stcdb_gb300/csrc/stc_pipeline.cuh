// Device buffers of one pipeline context and the per-step launchers.
#pragma once
#include "stc_common.cuh"
#include "stc_rules.cuh"
#include "stc_schema.cuh"

namespace stc {

constexpr uint32_t STRIPS_MAX = 64;     // horizontal strips of a leaf
constexpr uint32_t STRIP_STRIDE = 68;   // words of a leaf's strip starts (STRIPS_MAX + 1, padded)
constexpr uint32_t XSORT_MAX = 128;     // strips of at most this many members are in longitude order
constexpr uint32_t LEAF_SMALL = 256;    // kept members of the leaves k_leaf_small takes
constexpr uint32_t JOB_OWN = 1u << 31;

// A leaf as the refinement sees it.
struct __align__(16) LeafGeo {
  double lo_x, lo_y;       // low corner
  float inv, wx;           // strips per degree of latitude from the low edge; longitude window in degrees
  uint32_t strips;
  float ext_x, ext_y;      // extent in degrees
  uint32_t base, n;        // its members: spts[base .. base + n)
  uint32_t pad;
};

// counters of a step (PipeDev::ctr)
constexpr uint32_t MAX_SLICES = 64;  // of a long step kernel (stc_config.step_slices)
enum { CTR_MEMBERS = 0, CTR_SMALL, CTR_BIG, CTR_EXTRA, CTR_UNITS, CTR_POOL, CTR_JOBS, CTR_COUNT = CTR_JOBS + MAX_SLICES };

// Candidate positions per refinement job and lane: a row block's candidate
// ranges are cut into chunks of this many, so that the n^2 / 2 pair tests of
// a dense leaf spread over many warps.
constexpr uint32_t REFINE_CHUNK_DEFAULT = 256;  // tile length before the first step's density is known
// of dense leaves, of few rows, of few rows with few tests (choose_refine_chunk)
constexpr uint32_t REFINE_CHUNK_DENSE = 64, REFINE_CHUNK_FEW = 32, REFINE_CHUNK_FEWEST = 16;

struct PipeDev {
  // sizes
  uint32_t N, leaf_cap, G, S;
  unsigned long long B;            // meeting table slots
  unsigned long long B_magic;      // ceil(2^64 / B) for fast_mod
  unsigned long long C;            // candidate set slots (power of two)
  unsigned long long cand_cap;     // candidate list capacity
  unsigned long long E;            // emit buffer capacity
  unsigned long long U_cap;        // border units (refine_size*N - N - 1)
  // parameters
  double reach, x_buffer, y_buffer;
  float reach_f, x_buffer_f, y_buffer_f;
  double map_lo_x, map_lo_y, map_hi_x, map_hi_y;
  float fmap_lo_x, fmap_lo_y, fmap_hi_x, fmap_hi_y;  // float f: f >= map_lo <=> f >= fmap_lo, etc.
  uint32_t min_meet_time, grid_capacity, delay;
  int mbr_filter;
  uint32_t slices;                 // launches per long step kernel (stc_config.step_slices)
  uint32_t job_chunk;              // refinement jobs a warp takes at a time (stc_config.job_chunk)
  uint32_t general;                // 1: this step takes the general path, whatever its tiles (PathChoice)
  uint32_t job_share;              // 1: or one at a time from a common counter (job_shares)
  uint32_t refine_chunk;               // candidate positions per refinement job (16 or a multiple of 32)
  uint32_t refine_bps, hits_bps;   // blocks per SM of the pair tests (0: step_pairs chooses) and of the table update
  // state
  DevState *st;
  SchemaDev sd;
  SchemaWork sw;
  const double2 *xy;               // positions of the current step
  const double2 *xy_in = nullptr;  // when set: page-locked host positions the descent reads and
                                   // copies to xy (a buffer of the context's own)
  // partition
  unsigned long long *ctr;              // CTR_COUNT
  uint32_t *leaf_gid, *lastvalid;       // N
  uint32_t *rank;                       // N: the object's number within its leaf (any order)
  uint32_t *lpid, *lpid2;               // N: leaf member lists; the kept members of overfull leaves
  uint32_t *grid_count, *grid_start;    // G: members of each leaf, start of its list
  uint32_t *leaf_list;                  // leaves with members: small ones from the front, big from the end
  uint32_t leaves_max;                  // its length
  float4 *pts;                          // N: big leaves' members before the strip order
  float2 *sfxy;                         // N in strip order (as spts): float lon, lat of each member
  // each leaf's kept members, ordered by horizontal strip (strips at least
  // reach tall) and, within a small strip, by longitude: spts = leaf offsets
  // lx, ly, metres per degree of longitude, pid bits; scand = the member's
  // candidate ranges within the leaf: [i + 1, x & 0xFFFF) in its strip and
  // [x >> 16, y) in the next; sstart[g * STRIP_STRIDE + s] = first member of
  // strip s
  float4 *spts;
  uint2 *scand;
  uint16_t *sstart;
  LeafGeo *lgeo;                        // G
  // refinement jobs: (leaf, row block | JOB_OWN, first chunk, chunks)
  uint4 *jobs;
  unsigned long long jobs_extra;        // jobs beyond one per row block the list has room for
  uint32_t order_shift;                 // a hit's priority: unit rank << order_shift | member pid
  // border units
  uint32_t *bcount, *boff;              // N (border units per pid, their place in rank order)
  uint32_t *bsum;                       // units before each block of border_tile pids
  uint32_t border_tile;                 // 256 or 1024 pids per block of the border lookup
  uint32_t *bres;                       // 4N: first four lookup results per border point
  float border_delta;                   // fp32 band (metres) of the border lookup pre-filter
  float border_eps;                     // fp32 band (degrees) of its leaf test
  uint32_t *bu_gid, *bu_pid;            // U_cap (rank order)
  uint32_t *bu_rank, *bu_sorted_pos;    // U_cap: number within the leaf; places grouped by leaf
  uint32_t *bu_cnt, *bu_start;          // G
  // meetings
  Slot *slots;                          // B
  // hits of the step, binned by table tile (tile_of): bin j holds
  // min(bin_cnt[j], bin_cap) records, at hit_place; a hit its bin has no room
  // for is applied inside the pair tests
  HitRec *hits;                         // hit_records(nb, bin_cap)
  unsigned long long *hit_bounds;       // [MAX_SLICES + 1]: end of each part's hits (general steps)
  uint32_t nb, bin_cap;                 // tiles of the table, records per bin
  unsigned long long nb_magic;          // ceil(2^64 / nb)
  uint32_t *bin_cnt;                    // nb
  uint32_t *tile_live;                  // nb: occupied slots of each tile after the last step
  uint32_t *occ;                        // nb x OCC_WORDS: which ones, a bit a slot of the tile
  uint32_t runs;                        // runs of tiles the tiled update is cut into
  uint32_t *carry, *carry_cnt;          // runs x TILE_LOAD, runs: hits carried into each run
  Cand *cset;                           // C
  uint32_t *cand_list;                  // cand_cap
  stc_meeting *emit;                    // E
};

// Place of record i of bin j: bins are cut into chunks of HIT_CHUNK (16) records, the
// first chunks of all bins come first, then the second ones. The bins fill at
// much the same pace, so the step writes to a few hundred MB at a time and not
// to all of the buffer: scattered stores are bound by the reach of the address
// translation (67.7M records into 349526 bins, with their counters: 36 G/s bin
// after bin, 2.8 GB; 52 with chunks of 16; 80 if all went to 180 MB).
__host__ __device__ __forceinline__ unsigned long long hit_place(const PipeDev &p, uint32_t j, uint32_t i) {
  return ((unsigned long long)(i / HIT_CHUNK) * p.nb + j) * HIT_CHUNK + i % HIT_CHUNK;
}
__host__ __device__ __forceinline__ size_t hit_records(uint32_t nb, uint32_t bin_cap) {
  return (size_t)nb * ((bin_cap + HIT_CHUNK - 1) / HIT_CHUNK * HIT_CHUNK);
}

// Blocks an SM of the pair tests: three for each that it holds at once where
// the last warps are a larger part of the time (few rows, short tiles: 300k
// objects, half of them in hotspots, 0.46 -> 0.43 ms a step), else two.
constexpr uint32_t REFINE_THREADS = 256;
inline uint32_t refine_blocks(const PipeDev &p) {
  return p.refine_bps ? p.refine_bps : p.refine_chunk <= REFINE_CHUNK_FEW ? 12u : REFINE_BPS_BUILTIN;
}

// Whether warps take their jobs one by one from a common counter: `jobs` to
// take by `warps`. Dense leaves lie together, and with all jobs dealt out
// beforehand a fifth of the SMs' time was the wait for the last warps; asking
// costs more than that where a warp has few jobs, or a dozen short ones (long
// tiles: few candidates a job). ms of pair tests, dealt out and by demand: 10M
// uniform (47 jobs a warp) 2.38, 2.13; hotspot-1M (short tiles) 1.40, 1.22; the
// stress model 1.89, 1.66; 3M uniform (14 jobs a warp) 0.28, 0.31; 60k in
// hotspots 0.119, 0.126.
inline bool job_shares(unsigned long long jobs, unsigned long long warps, uint32_t chunk) {
  return jobs >= (chunk <= REFINE_CHUNK_DENSE ? 8ull : 24ull) * warps;
}

// stc_partition.cu
// the descent (leaf of every object), the leaves' members in strip order with
// their jobs, and beside those the border units with theirs
void step_descend(PipeDev &p, cudaStream_t s);
void step_leaves(PipeDev &p, cudaStream_t s);
void step_border(PipeDev &p, cudaStream_t s);
// stc_refine.cu
// the pair tests, which bin the step's hits by table tile, and the general
// path's table update of them (nothing when the tiled path took the step)
void step_pairs(PipeDev &p, cudaStream_t s);
void step_hits(PipeDev &p, cudaStream_t s);
// of a step told to be general: part `part` of `parts` of the pair tests, whose
// hits go to the buffer in sequence, and the table update of them, which may
// run beside the next part
constexpr uint32_t GENERAL_PARTS = 4;  // or more, for step_slices
void step_pairs_part(PipeDev &p, uint32_t part, uint32_t parts, cudaStream_t s);
void step_hits_part(PipeDev &p, uint32_t part, cudaStream_t s);
// stc_table.cu: the tiled table update and sweep. plan decides whether the
// step takes it and finds what is carried into each run of tiles.
constexpr uint32_t OCC_WORDS = TILE_SLOTS / 32;
cudaError_t table_prepare();
void table_sizes(PipeDev &p);           // nb and runs of a table of p.B slots
void count_tiles(PipeDev &p, cudaStream_t s);
void unpack_tiles(PipeDev &p, uint32_t layout, cudaStream_t s);  // every meeting into its slot
void step_table_slots(PipeDev &p, cudaStream_t s);  // the same if the tiles are packed
void step_table_plan(PipeDev &p, cudaStream_t s);
void step_table(PipeDev &p, cudaStream_t s);
// stc_meetings.cu: the general path's insert and sweep
void step_insert(PipeDev &p, cudaStream_t s);
void step_sweep(PipeDev &p, cudaStream_t s);
void init_tables(PipeDev &p, cudaStream_t s);
void step_begin(PipeDev &p, const uint32_t *t_pinned, cudaStream_t s);

}  // namespace stc
