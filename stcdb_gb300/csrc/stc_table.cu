// Step kernel (c), tiled: the table update, the ordered insertion of new
// meetings and the expire/emit sweep in one pass over the meeting table.
// Before and after, one GB300, per step: 10M uniform objects (2^28 slots,
// 67.7M hits, 36.7M of them new) 8.4 ms of pair tests with the update beside
// them and 2.7 of sweep -> 2.0 ms of pair tests and 2.6 of k_table;
// hotspot-1M (34.7M hits) 4.0 + 1.9 -> 1.15 + 1.6 ms. Bound by instruction
// issue (60% of the slots in a tile's chain of short phases; DRAM at 30%).
//
// The pair tests leave the step's hits binned by table tile (TILE_SLOTS
// slots, about; stc_refine.cu). A block takes a run of consecutive tiles and,
// tile by tile, copies the tile's keys to shared memory, applies the tile's
// hits to it there (extensions, and claims of empty slots by priority), then
// finalises claims, drops or emits ended meetings and writes what goes on.
// Applying the hits one by one at random over the table and sweeping it
// afterwards brought a 128-byte line from DRAM for every hit and the whole
// table again for the sweep; this way the table streams through once.
//
// Only meetings stream: the tiled update leaves each tile packed, its
// meetings in slot order at one end of the tile, their slots in a bit a slot
// (PipeDev::occ), and reads it so in the next step, writing to the other end.
// Tables are sized for the worst hour and mostly empty (hotspot-1M: 35M
// meetings in 2^28 slots), and meetings in their slots cost DRAM its 64-byte
// atoms and L2 a 32-byte sector each: 268M slots at a density of 0.2 took 1.50
// ms to read and write back slot by slot, 0.58 packed. k_table, all slots read
// -> occupied ones read in place -> packed: hotspot-1M 2.26 -> 2.35 -> 1.88 ms,
// 10M 3.0 -> 3.2 -> 2.5. The general path works on slots: k_table_halo puts
// the meetings of a step that needs it into theirs first (tile_unpack).
//
// A hit whose probe walk passes the end of its tile is carried to the next
// tile of the run. What the last tiles before a run would carry into it is
// found first, by k_table_halo: it works through the `halo` tiles before each
// run, entering them with nothing carried, and keeps only what comes out.
//
// Why that is exact. Let c be the largest (occupied slots + binned hits) of
// any tile, T the smallest tile. A key never walks past a slot that stays
// empty. If c < T, no tile passes more than c keys on: a tile with a slot
// that stays empty passes on only keys homed behind it, at most its own
// hits; a full tile passes on at most what it receives, less T - c (extended
// hits and filled slots are no longer carried), and not all tiles are full.
// So the halo's tiles end up with at most c * halo slots of their own and c
// of those carried in: if c * (halo + 1) < halo * T, at least one slot s of
// the halo stays empty, nothing carried into the halo passes s, and what
// leaves the halo is decided by keys homed behind s. Taking keys away from
// an insertion by priority moves no other key further, so s stays empty in
// the halo run on its own and the keys behind it end up in the same slots.
// The rule is checked on the device before anything is written (fuse_halo);
// a step that fails it (a loaded table, or more hits in a bin than it holds)
// takes the general path: k_hits, k_insert_ordered and k_sweep. The steps after
// it are told to beforehand until the tiles would do again (PathChoice).
//
// Claims by priority in shared memory are the deferred acceptance of
// stc_insert.cuh: an empty slot's start word names the hit claiming it (its
// record's place counted from the run's first bin), a hit of lower priority
// evicts it and carries the evicted one on, so the outcome is the one of
// sequential insertion in priority order, whatever the timing.
#include <algorithm>

#include "stc_insert.cuh"

namespace stc {

namespace {

constexpr uint32_t TB_THREADS = 128;
constexpr uint32_t TB_BLOCKS_PER_SM = 8;
constexpr uint32_t TB_WAVES = 5;        // runs are short, so that query batches get SMs between them
constexpr uint32_t TB_RUN_TILES = 16;   // shortest run worth its halo, where the table has that many tiles
constexpr uint32_t TB_RECS = 256;       // hits whose pair and order are held in shared memory
constexpr uint32_t TB_STAGE = 48;       // emitted meetings staged per block
constexpr uint32_t TB_DUPS = 64;        // hits of possible double pairs listed per tile

// 27.5 KB, eight blocks an SM with no byte to spare: a tile is a chain of short phases of a hundred or
// two items each, so many blocks of few warps keep the SM busy. It holds what
// the phases look up at random, the keys and each hit's pair and order; boxes
// and start times stay in global memory (L2 by then) until the write-back
// (loading them ahead and keeping the hits' boxes here, with seven blocks:
// the same time).
struct __align__(128) Tile {
  unsigned long long key[TILE_SLOTS];
  ulonglong2 rec[TB_RECS];              // (pair, order) of the tile's hits, then of those carried in
  uint32_t mark[TILE_SLOTS];            // the hit that extends the meeting or claims the empty slot; STC_NONE
  uint32_t carry[2][TILE_LOAD];         // hits carried in and out: places counted from the run's first bin
  stc_meeting stage[TB_STAGE];
  uint32_t fresh[2 * TILE_LOAD];        // hits without a meeting: number | first empty slot << 16
  uint32_t dup[TB_DUPS];                // the same of possibly double ones
  uint16_t list[TILE_SLOTS];            // the slots in use: the tile's occupied ones, then those claimed
  uint32_t bits[OCC_WORDS];             // occupied slots of the tile
  uint32_t left[OCC_WORDS];             // slots that stay occupied after the step
  unsigned long long base;              // emit position of a staged batch
  // counters in turns, so that one is reset while its neighbours are in use
  uint32_t ncarry[3], ndup[2], nnew[2], nlist[2], nstage;
};

// Record `id` of a run whose bins are counted from tile r0 (cyclic).
__device__ __forceinline__ const HitRec *run_record(const PipeDev &p, uint32_t r0, uint32_t id) {
  const uint32_t seq = id / p.bin_cap;
  uint32_t tile = r0 + seq;
  if (tile >= p.nb) tile -= p.nb;
  return p.hits + hit_place(p, tile, id - seq * p.bin_cap);
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// First record of the n meetings of a packed tile, counted from its start.
__device__ __forceinline__ uint32_t packed_at(uint32_t layout, uint32_t len, uint32_t n) {
  return layout == TABLE_BACK ? len - n : 0u;
}

// Starts the copies of a tile's hits (pair and order) and meetings (keys, each
// to its slot; listed from s.bits) to shared memory, where every other slot is
// empty; returns how many meetings there are. Called by the whole block,
// before the barrier that opens tile_apply.
__device__ __forceinline__ uint32_t tile_fetch(const PipeDev &p, Tile &s, uint32_t tile, unsigned long long start,
                                               uint32_t len, uint32_t n, uint32_t turn, uint32_t layout) {
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  for (uint32_t i = threadIdx.x; i < min(n, TB_RECS); i += TB_THREADS)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(&s.rec[i])), "l"(p.hits + hit_place(p, tile, i)) : "memory");
  const uint32_t w = lane < OCC_WORDS ? s.bits[lane] : 0u;
  uint32_t incl = __popc(w);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
    if ((int)lane >= d) incl += up;
  }
  const uint32_t held = __shfl_sync(0xffffffffu, incl, 31), front = packed_at(layout, len, held);
  if (threadIdx.x == 0) s.nlist[turn & 1u] = held;
#pragma unroll
  for (uint32_t j0 = 0; j0 < OCC_WORDS; j0 += TB_THREADS / 32) {  // a word a warp, a slot a lane
    const uint32_t j = j0 + warp;
    const uint32_t word = __shfl_sync(0xffffffffu, w, j), upto = __shfl_sync(0xffffffffu, incl, j);
    if ((word >> lane) & 1u) {
      const uint32_t i = j * 32u + lane, x = upto - __popc(word >> lane);
      s.list[x] = (uint16_t)i;
      const Slot *from = p.slots + start + (layout == TABLE_SLOTS ? i : front + x);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(&s.key[i])), "l"(&from->key) : "memory");
    }
  }
  return held;
}

__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void slot_clear(Tile &s, uint32_t i) {
  s.key[i] = STC_EMPTY_KEY;
  s.mark[i] = STC_NONE;
}

__device__ __forceinline__ uint32_t bin_hits(const PipeDev &p, uint32_t tile) {
  return min(p.bin_cnt[tile], p.bin_cap);
}

// The tile being worked on, as every thread sees it.
struct TileView {
  unsigned long long start;  // its first slot
  uint32_t tile;
  uint32_t n, nc;            // its hits, hits carried in
  uint32_t r0, id0;          // the run's first bin, the place of this bin's first hit
  uint32_t len, turn;        // slots, the tile's number in its run
};

// Record of hit i of the tile (i < n: its own, then the ones carried in).
__device__ __forceinline__ const HitRec *tile_rec(const PipeDev &p, const Tile &s, const TileView &v, uint32_t i) {
  return i < v.n ? p.hits + hit_place(p, v.tile, i) : run_record(p, v.r0, s.carry[v.turn & 1u][i - v.n]);
}

// Its pair (a | b << 32) and order.
__device__ __forceinline__ ulonglong2 tile_pair(const PipeDev &p, const Tile &s, const TileView &v, uint32_t i) {
  if (i < TB_RECS) return s.rec[i];
  return __ldg((const ulonglong2 *)tile_rec(p, s, v, i));
}

__device__ __forceinline__ unsigned long long pair_key(unsigned long long ab) {
  return stc_cantor((uint32_t)ab, (uint32_t)(ab >> 32));
}

// First slot at or behind `pos` that holds `key` or is empty; v.len if none.
__device__ __forceinline__ uint32_t tile_probe(const Tile &s, const TileView &v, unsigned long long key, uint32_t pos,
                                               bool &found) {
  unsigned long long k = STC_EMPTY_KEY;
  for (; pos < v.len; pos++) {
    k = s.key[pos];  // keys do not change while hits are applied
    if (k == key || k == STC_EMPTY_KEY) break;
  }
  found = pos < v.len && k == key;
  return pos;
}

// Slot pos is occupied after the step.
__device__ __forceinline__ void tile_stays(Tile &s, uint32_t pos) { atomicOr(&s.left[pos >> 5], 1u << (pos & 31u)); }

// Hit i, which found no meeting before slot `pos` (empty, or the tile's
// end): claims an empty slot, carrying on whatever it evicts; ends at a
// meeting of its own behind an empty slot it lost; or leaves the tile.
__device__ __forceinline__ void tile_claim(const PipeDev &p, Tile &s, const TileView &v, uint32_t i, uint32_t pos) {
  const ulonglong2 h = tile_pair(p, s, v, i);
  unsigned long long key = pair_key(h.x), prio = h.y & ~DUP_BIT;
  bool found = false;
  for (;;) {
    if (pos >= v.len) {
      const uint32_t c = atomicAdd(&s.ncarry[(v.turn + 1) % 3], 1u);
      if (c < TILE_LOAD)
        s.carry[(v.turn & 1u) ^ 1u][c] = i < v.n ? v.id0 + i : s.carry[v.turn & 1u][i - v.n];
      else
        stc_set_error(p.st, ERR_PROBE, c);  // never, by fuse_halo's rule
      return;
    }
    uint32_t *w = &s.mark[pos];
    if (found) {  // extends its own meeting (both instances of a double pair may: the same box)
      *w = i;
      tile_stays(s, pos);
      return;
    }
    uint32_t cur = atomicCAS(w, STC_NONE, i);
    if (cur == STC_NONE) {  // settled: a new meeting
      s.list[atomicAdd(&s.nlist[v.turn & 1u], 1u)] = (uint16_t)pos;
      tile_stays(s, pos);
      return;
    }
    for (;;) {  // a claimed slot stays claimed
      const ulonglong2 o = tile_pair(p, s, v, cur);
      const unsigned long long other = o.y & ~DUP_BIT;
      if (prio > other) break;  // lost this slot
      const uint32_t old = atomicCAS(w, cur, i);
      if (old == cur) {  // carry the evicted hit onward
        i = cur;
        key = pair_key(o.x);
        prio = other;
        break;
      }
      cur = old;
    }
    pos = tile_probe(s, v, key, pos + 1, found);
  }
}

// Applies the hits of a tile and the ones carried into it to its slots in
// shared memory, whose copies have been started: afterwards every hit has
// marked its meeting, claimed an empty slot or been put on the other carry
// list. First every hit looks its meeting up, then the ones without one,
// packed together, claim slots: the two loops diverge little, where one loop
// for both had every warp wait for its longest chain of claims. Ends with the
// block's barrier.
__device__ __forceinline__ void tile_apply(const PipeDev &p, Tile &s, const TileView &v) {
  const uint32_t tid = threadIdx.x, lt_mask = (1u << lane_id()) - 1u, par = v.turn & 1u;
  for (uint32_t i = tid; i < v.nc; i += TB_THREADS)
    if (v.n + i < TB_RECS) s.rec[v.n + i] = __ldg((const ulonglong2 *)run_record(p, v.r0, s.carry[par][i]));
  fetch_wait();
  __syncthreads();
  const uint32_t total = v.n + v.nc;
  for (uint32_t i0 = tid & ~31u; i0 < total; i0 += TB_THREADS) {
    const uint32_t i = i0 + lane_id();
    bool claims = false;
    uint32_t pos = 0;
    if (i < total) {
      const ulonglong2 h = tile_pair(p, s, v, i);
      const unsigned long long key = pair_key(h.x);
      if (i < v.n) pos = (uint32_t)(fast_mod(key, p.B, p.B_magic) - v.start);
      bool found;
      pos = tile_probe(s, v, key, pos, found);
      if (found) {
        s.mark[pos] = i;
        tile_stays(s, pos);
      } else if (i < v.n && (h.y & DUP_BIT)) {  // the pair's other instance decides which one claims
        const uint32_t d = atomicAdd(&s.ndup[par], 1u);
        if (d < TB_DUPS) s.dup[d] = i | pos << 16;
      } else {
        claims = true;
      }
    }
    const uint32_t ball = __ballot_sync(0xffffffffu, claims);
    if (ball) {
      uint32_t at = 0;
      if (lane_id() == 0) at = atomicAdd(&s.nnew[par], (uint32_t)__popc(ball));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(ball & lt_mask);
      if (claims) s.fresh[at] = i | pos << 16;
    }
  }
  __syncthreads();
  const uint32_t m = s.nnew[par];
  for (uint32_t x = tid; x < m; x += TB_THREADS) tile_claim(p, s, v, s.fresh[x] & 0xFFFFu, s.fresh[x] >> 16);
  // hits flagged as possibly double: a pair's instances are in one bin, and
  // the one of lowest priority claims for all
  const uint32_t nd = s.ndup[par];
  if (nd) {
    const bool listed = nd <= TB_DUPS;
    for (uint32_t x = tid; x < (listed ? nd : v.n); x += TB_THREADS) {
      const uint32_t i = listed ? s.dup[x] & 0xFFFFu : x;
      const ulonglong2 h = tile_pair(p, s, v, i);
      if (!(h.y & DUP_BIT)) continue;
      bool first = true;
      for (uint32_t y = 0; y < (listed ? nd : v.n) && first; y++) {
        const ulonglong2 o = tile_pair(p, s, v, listed ? s.dup[y] & 0xFFFFu : y);
        if (o.x == h.x && (o.y & DUP_BIT) && o.y < h.y) first = false;
      }
      if (!first) continue;
      uint32_t pos = s.dup[x & (TB_DUPS - 1)] >> 16;
      if (!listed) {
        const unsigned long long key = pair_key(h.x);
        bool found;
        pos = tile_probe(s, v, key, (uint32_t)(fast_mod(key, p.B, p.B_magic) - v.start), found);
        if (found) continue;  // extended already
      }
      tile_claim(p, s, v, i, pos);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void load_slot(const Slot *d, ulonglong2 &key_times, float4 &box) {
  uint32_t r[8];
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(d)
               : "memory");
  key_times = make_ulonglong2(r[0] | (unsigned long long)r[1] << 32, r[2] | (unsigned long long)r[3] << 32);
  box = make_float4(__uint_as_float(r[4]), __uint_as_float(r[5]), __uint_as_float(r[6]), __uint_as_float(r[7]));
}

// One 32-byte store: a whole sector, written once and read next step.
__device__ __forceinline__ void store_slot(Slot *d, unsigned long long key, uint32_t start, uint32_t end, float4 m) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(d), "r"((uint32_t)key),
               "r"((uint32_t)(key >> 32)), "r"(start), "r"(end), "r"(__float_as_uint(m.x)),
               "r"(__float_as_uint(m.y)), "r"(__float_as_uint(m.z)), "r"(__float_as_uint(m.w))
               : "memory");
}

// Tiles of run r of `runs`: [r * nb / runs, (r + 1) * nb / runs).
__device__ __forceinline__ uint32_t run_start(const PipeDev &p, uint32_t r) {
  return (uint32_t)((unsigned long long)r * p.nb / p.runs);
}

// The meetings of a packed tile into their slots; slots: shared memory for
// TILE_SLOTS of them. Called by the whole block.
__device__ void tile_unpack(const PipeDev &p, Slot *slots, uint32_t tile, uint32_t layout) {
  const unsigned long long start = tile_start(p, tile);
  const uint32_t len = (uint32_t)(tile_start(p, tile + 1) - start), lane = lane_id();
  const uint32_t w = lane < OCC_WORDS ? p.occ[(size_t)tile * OCC_WORDS + lane] : 0u;
  uint32_t incl = __popc(w);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
    if ((int)lane >= d) incl += up;
  }
  const uint32_t held = __shfl_sync(0xffffffffu, incl, 31);
  const Slot *from = p.slots + start + packed_at(layout, len, held);
  for (uint32_t x = threadIdx.x; x < held; x += blockDim.x) slots[x] = from[x];
  __syncthreads();
  for (uint32_t i0 = threadIdx.x & ~31u; i0 < len; i0 += blockDim.x) {
    const uint32_t i = i0 + lane, word = __shfl_sync(0xffffffffu, w, i0 >> 5);
    const uint32_t upto = __shfl_sync(0xffffffffu, incl, i0 >> 5);
    if (i >= len) continue;
    Slot d = {STC_EMPTY_KEY, STC_NONE, STC_NONE, STC_INIT_LO, STC_INIT_LO, STC_INIT_HI, STC_INIT_HI};
    if ((word >> lane) & 1u) d = slots[upto - __popc(word >> lane)];
    store_slot(&p.slots[start + i], d.key, d.start, d.end, make_float4(d.lo_x, d.lo_y, d.hi_x, d.hi_y));
  }
  __syncthreads();
}

}  // namespace

// The largest bin and the largest (occupied slots + hits) of a tile, which
// decide the step's path (fuse_halo). A step told to be general has no bins:
// the load is the meetings of the step before (PathChoice), if it counted them.
__global__ void __launch_bounds__(256) k_table_plan(PipeDev p) {
  after_previous();
  const uint32_t told = p.st->told;
  uint32_t load = 0, most = 0;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < p.nb; j += gridDim.x * blockDim.x) {
    const uint32_t c = p.bin_cnt[j];
    most = max(most, c);
    load = max(load, c + p.tile_live[j]);
  }
  if (told & TOLD_STALE) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicMax(&p.st->tile_load, (unsigned long long)LOAD_UNKNOWN);
    load = 0;
  }
  load = __reduce_max_sync(0xffffffffu, load);
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane_id() == 0) {
    if (load) atomicMax(&p.st->tile_load, (unsigned long long)load);
    if (most) atomicMax(&p.st->hit_max, (unsigned long long)most);
  }
}

// What is carried into each run: the halo tiles before it, worked through
// with nothing carried into them. Writes nothing but the carry lists.
__global__ void __launch_bounds__(TB_THREADS, TB_BLOCKS_PER_SM) k_table_halo(PipeDev p) {
  after_previous();
  extern __shared__ __align__(128) unsigned char smem[];
  Tile &s = *(Tile *)smem;
  const uint32_t halo = fuse_halo(p), layout = p.st->packed;
  if (!halo) {
    if (layout != TABLE_SLOTS)
      for (uint32_t tile = blockIdx.x; tile < p.nb; tile += gridDim.x) tile_unpack(p, (Slot *)smem, tile, layout);
    return;
  }
  const uint32_t tid = threadIdx.x;
  const uint32_t r = blockIdx.x;
  const uint32_t first = run_start(p, r), r0 = first >= halo ? first - halo : first + p.nb - halo;
  TileView v;
  v.r0 = r0;
  for (uint32_t i = tid; i < TILE_SLOTS; i += TB_THREADS) slot_clear(s, i);
  if (tid == 0) {
    s.ncarry[0] = s.ncarry[1] = s.ncarry[2] = s.ndup[0] = s.ndup[1] = s.nnew[0] = s.nnew[1] = 0;
  }
  __syncthreads();
  for (uint32_t q = 0; q < halo; q++) {
    const uint32_t tile = r0 + q >= p.nb ? r0 + q - p.nb : r0 + q;
    v.turn = q;
    v.start = tile_start(p, tile);
    v.len = (uint32_t)(tile_start(p, tile + 1) - v.start);
    v.n = bin_hits(p, tile);
    v.nc = min(s.ncarry[q % 3], TILE_LOAD);
    v.id0 = q * p.bin_cap;
    v.tile = tile;
    if (tid < OCC_WORDS) s.bits[tid] = p.occ[(size_t)tile * OCC_WORDS + tid];
    __syncthreads();
    tile_fetch(p, s, tile, v.start, v.len, v.n, q, layout);
    tile_apply(p, s, v);
    const uint32_t used = s.nlist[q & 1u];
    for (uint32_t x = tid; x < used; x += TB_THREADS) slot_clear(s, s.list[x]);
    if (tid == 0) s.ncarry[(q + 2) % 3] = s.ndup[(q & 1u) ^ 1u] = s.nnew[(q & 1u) ^ 1u] = 0;
    __syncthreads();
  }
  const uint32_t n = min(s.ncarry[halo % 3], TILE_LOAD);
  for (uint32_t i = tid; i < n; i += TB_THREADS) p.carry[(size_t)r * TILE_LOAD + i] = s.carry[halo & 1u][i];
  if (tid == 0) p.carry_cnt[r] = n;
}

// One block per run. Part `part` of `parts` works runs
// [runs * part / parts, runs * (part + 1) / parts).
__global__ void __launch_bounds__(TB_THREADS, TB_BLOCKS_PER_SM) k_table(PipeDev p, uint32_t part, uint32_t parts) {
  after_previous();
  extern __shared__ __align__(128) unsigned char smem[];
  Tile &s = *(Tile *)smem;
  const uint32_t halo = fuse_halo(p), layout = p.st->packed;
  if (!halo) return;
  const uint32_t into = layout == TABLE_FRONT ? TABLE_BACK : TABLE_FRONT;
  const bool same_t = p.st->same_t != 0;
  const uint32_t t = p.st->step_t, tid = threadIdx.x, lane = lane_id();
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t q0 = (uint32_t)((unsigned long long)p.runs * part / parts);
  const uint32_t q1 = (uint32_t)((unsigned long long)p.runs * (part + 1) / parts);
  const uint32_t r = q0 + blockIdx.x;
  if (r >= q1) return;
  const uint32_t first = run_start(p, r), last = run_start(p, r + 1);
  uint32_t active = 0, fresh = 0, emitted = 0;
  TileView v;
  v.r0 = first >= halo ? first - halo : first + p.nb - halo;
  v.start = tile_start(p, first);
  v.len = (uint32_t)(tile_start(p, first + 1) - v.start);
  v.n = bin_hits(p, first);
  const uint32_t nc = min(p.carry_cnt[r], TILE_LOAD);
  for (uint32_t i = tid; i < nc; i += TB_THREADS) s.carry[0][i] = p.carry[(size_t)r * TILE_LOAD + i];
  for (uint32_t i = tid; i < TILE_SLOTS; i += TB_THREADS) slot_clear(s, i);
  if (tid < OCC_WORDS) {
    s.bits[tid] = p.occ[(size_t)first * OCC_WORDS + tid];
    s.left[tid] = same_t ? s.bits[tid] : 0u;
  }
  if (tid == 0) {
    s.ncarry[0] = nc;
    s.ncarry[1] = s.ncarry[2] = s.ndup[0] = s.ndup[1] = s.nnew[0] = s.nnew[1] = s.nstage = 0;
  }
  __syncthreads();
  uint32_t held = tile_fetch(p, s, first, v.start, v.len, v.n, 0, layout);
  for (uint32_t tile = first; tile < last; tile++) {
    v.turn = tile - first;
    v.id0 = (halo + v.turn) * p.bin_cap;
    v.tile = tile;
    v.nc = min(s.ncarry[v.turn % 3], TILE_LOAD);
    // the next tile's count and occupied slots, on their way beside the hits
    const uint32_t next_n = tile + 1 < last ? bin_hits(p, tile + 1) : 0u;
    uint32_t next_bits = 0;
    if (tid < OCC_WORDS && tile + 1 < last) next_bits = p.occ[(size_t)(tile + 1) * OCC_WORDS + tid];
    tile_apply(p, s, v);
    // write what stays, packed; emit what ended (tracing/meeting.cpp:47-67)
    const uint32_t used = s.nlist[v.turn & 1u];
    const uint32_t left = lane < OCC_WORDS ? s.left[lane] : 0u;
    uint32_t incl = __popc(left);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
      if ((int)lane >= d) incl += up;
    }
    const uint32_t stay = __shfl_sync(0xffffffffu, incl, 31);
    const Slot *const from = p.slots + v.start + packed_at(layout, v.len, held);
    Slot *const to = p.slots + v.start + packed_at(into, v.len, stay);
    // old and new records lie at opposite ends of the tile; where they would
    // meet, and where the old ones are still in their slots, all are read
    // before any is written
    const bool tight = layout == TABLE_SLOTS || held + stay > v.len;
    ulonglong2 kept[(TILE_LOAD + TB_THREADS - 1) / TB_THREADS];
    float4 kept_box[(TILE_LOAD + TB_THREADS - 1) / TB_THREADS];
    if (tight) {
#pragma unroll 1
      for (uint32_t x = tid, u = 0; x < held; x += TB_THREADS, u++)
        load_slot(layout == TABLE_SLOTS ? p.slots + v.start + s.list[x] : from + x, kept[u], kept_box[u]);
      __syncthreads();
    }
#pragma unroll 1
    for (uint32_t x0 = tid & ~31u, u = 0; x0 < used; x0 += TB_THREADS, u++) {
      const uint32_t x = x0 + lane;
      bool emit = false;
      uint32_t i = 0;
      unsigned long long k = STC_EMPTY_KEY;
      ulonglong2 old = make_ulonglong2(STC_EMPTY_KEY, ~0ull);  // key; start and end times
      float4 box = make_float4(STC_INIT_LO, STC_INIT_LO, STC_INIT_HI, STC_INIT_HI);
      if (x < used) {
        i = s.list[x];
        k = s.key[i];
        if (x < held) {
          if (tight) {
            old = kept[u];
            box = kept_box[u];
          } else {
            load_slot(from + x, old, box);
          }
        }
      }
      const uint32_t rank = __shfl_sync(0xffffffffu, incl, i >> 5) -
                            __popc(__shfl_sync(0xffffffffu, left, i >> 5) >> (i & 31u));
      if (x < used) {
        const uint32_t h = s.mark[i];
        float4 m = box;
        if (h != STC_NONE) {
          // an extended meeting grows by both objects' positions
          // (tracing/refinement.cpp:40-42, MBR cuda/geometry.cu:474-478); a claim
          // becomes a new one (cuda/geometry.cu:480-489): start = end = t
          const float4 g = __ldg((const float4 *)&tile_rec(p, s, v, h)->lo_x);
          m = make_float4(fminf(box.x, g.x), fminf(box.y, g.y), fmaxf(box.z, g.z), fmaxf(box.w, g.w));
        }
        if (k == STC_EMPTY_KEY) {
          fresh++;
          store_slot(to + rank, pair_key(tile_pair(p, s, v, h).x), t, t, m);
        } else if (h != STC_NONE || same_t) {  // (with the last step's time again, all go on)
          store_slot(to + rank, k, (uint32_t)old.y, t, m);
        } else if (t - (uint32_t)old.y >= p.min_meet_time + 1) {
          emit = !p.mbr_filter ||
                 (box.x >= p.fmap_lo_x && box.z <= p.fmap_hi_x && box.y >= p.fmap_lo_y && box.w <= p.fmap_hi_y);
        }
        slot_clear(s, i);
      }
      const uint32_t ball = __ballot_sync(0xffffffffu, emit);
      if (ball) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(&s.nstage, (uint32_t)__popc(ball));
        b = __shfl_sync(0xffffffffu, b, 0) + __popc(ball & lt_mask);
        if (emit) {
          stc_meeting e;
          cantor_decode(k, &e.pid_lo, &e.pid_hi);
          e.start = (uint32_t)old.y;
          e.end = (uint32_t)(old.y >> 32);
          e.mbr[0] = box.x; e.mbr[1] = box.y; e.mbr[2] = box.z; e.mbr[3] = box.w;
          emitted++;
          if (b < TB_STAGE) {
            s.stage[b] = e;
          } else {
            const unsigned long long pos = agg_inc(&p.st->emit_count);
            if (pos < p.E) p.emit[pos] = e;
            else stc_set_error(p.st, ERR_EMIT, (uint32_t)min(pos - p.E, 0xFFFFFFFFull));
          }
        }
      }
    }
    if (tid < OCC_WORDS) s.bits[tid] = next_bits;
    if (tid == 0) {
      const uint32_t next = (v.turn & 1u) ^ 1u;
      s.ncarry[(v.turn + 2) % 3] = s.ndup[next] = s.nnew[next] = 0;
    }
    __syncthreads();
    const uint32_t staged = min(s.nstage, TB_STAGE);
    const bool flush = staged && (staged > TB_STAGE / 2 || tile + 1 == last);
    v.start += v.len;
    v.len = (uint32_t)(tile_start(p, min(tile + 2, p.nb)) - v.start);
    v.n = next_n;
    if (tid == 0 && flush) s.base = atomicAdd(&p.st->emit_count, (unsigned long long)staged);
    if (tid < OCC_WORDS) {
      s.left[tid] = same_t ? s.bits[tid] : 0u;
      p.occ[(size_t)tile * OCC_WORDS + tid] = left;
    }
    if (tid == 0) {
      p.tile_live[tile] = stay;
      active += stay;
    }
    if (tile + 1 < last) held = tile_fetch(p, s, tile + 1, v.start, v.len, next_n, v.turn + 1, layout);
    if (flush) {
      __syncthreads();
      const unsigned long long base = s.base;
      for (uint32_t i = tid; i < 2 * staged; i += TB_THREADS) {
        const unsigned long long pos = base + (i >> 1);
        if (pos < p.E) ((uint4 *)&p.emit[pos])[i & 1u] = ((const uint4 *)&s.stage[i >> 1])[i & 1u];
        else stc_set_error(p.st, ERR_EMIT, (uint32_t)min(pos - p.E, 0xFFFFFFFFull));
      }
      __syncthreads();
      if (tid == 0) s.nstage = 0;
      __syncthreads();
    }
  }
  active = __reduce_add_sync(0xffffffffu, active);
  fresh = __reduce_add_sync(0xffffffffu, fresh);
  emitted = __reduce_add_sync(0xffffffffu, emitted);
  if (lane == 0) {
    if (active) atomicAdd(&p.st->taken, (unsigned long long)active);
    if (fresh) atomicAdd(&p.st->fast_claims, (unsigned long long)fresh);
    if (emitted) atomicAdd(&p.st->step_emitted, (unsigned long long)emitted);
  }
}

// Occupied slots of every tile, from the table (after a restore).
__global__ void k_tile_count(PipeDev p) {
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.B;
       i += (unsigned long long)gridDim.x * blockDim.x)
    if (p.slots[i].key != STC_EMPTY_KEY) {
      const uint32_t tile = tile_of(p, i), at = (uint32_t)(i - tile_start(p, tile));
      atomicAdd(&p.tile_live[tile], 1u);
      atomicOr(&p.occ[(size_t)tile * OCC_WORDS + (at >> 5)], 1u << (at & 31u));
    }
}

static_assert(sizeof(Tile) + 1024 <= 228 * 1024 / TB_BLOCKS_PER_SM, "blocks per SM");
static_assert(sizeof(Tile) >= TILE_SLOTS * sizeof(Slot), "k_table_halo unpacks tiles in it");

cudaError_t table_prepare() {
  cudaError_t e = cudaFuncSetAttribute(k_table_halo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Tile));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_table, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Tile));
  return e;
}

void table_sizes(PipeDev &p) {
  p.nb = (uint32_t)((p.B + TILE_SLOTS - 1) / TILE_SLOTS);
  p.nb_magic = p.nb > 1 ? ~0ull / p.nb + 1 : 0;  // ceil(2^64 / nb) (nb = 1 never takes the tiled path)
  const uint32_t wave = (uint32_t)num_sms() * TB_BLOCKS_PER_SM;
  // at least two tiles a run: with one the halo is as long as the run, and the
  // few blocks that get two are waited for all the same
  p.runs = std::min(std::max(p.nb / 2, 1u), std::min(wave * TB_WAVES, std::max(wave, p.nb / TB_RUN_TILES)));
}

void count_tiles(PipeDev &p, cudaStream_t s) {
  cudaMemsetAsync(p.tile_live, 0, (size_t)p.nb * sizeof(uint32_t), s);
  cudaMemsetAsync(p.occ, 0, (size_t)p.nb * OCC_WORDS * sizeof(uint32_t), s);
  STC_KL k_tile_count<<<num_sms() * 8, 256, 0, s>>>(p);
}

__global__ void __launch_bounds__(TB_THREADS) k_table_unpack(PipeDev p, uint32_t layout) {
  __shared__ Slot slots[TILE_SLOTS];
  for (uint32_t tile = blockIdx.x; tile < p.nb; tile += gridDim.x) tile_unpack(p, slots, tile, layout);
  if (blockIdx.x == 0 && threadIdx.x == 0) p.st->packed = TABLE_SLOTS;
}

void unpack_tiles(PipeDev &p, uint32_t layout, cudaStream_t s) {
  STC_KL k_table_unpack<<<num_sms() * 8, TB_THREADS, 0, s>>>(p, layout);
}

__global__ void __launch_bounds__(TB_THREADS) k_table_slots(PipeDev p) {
  __shared__ Slot slots[TILE_SLOTS];
  const uint32_t layout = p.st->packed;
  if (layout == TABLE_SLOTS) return;
  for (uint32_t tile = blockIdx.x; tile < p.nb; tile += gridDim.x) tile_unpack(p, slots, tile, layout);
}
__global__ void k_layout_slots(DevState *st) { st->packed = TABLE_SLOTS; }

void step_table_slots(PipeDev &p, cudaStream_t s) {
  STC_KL k_table_slots<<<num_sms() * 8, TB_THREADS, 0, s>>>(p);
  STC_KL k_layout_slots<<<1, 1, 0, s>>>(p.st);
}

void step_table_plan(PipeDev &p, cudaStream_t s) {
  launch_behind(k_table_plan, std::min<unsigned>((p.nb + 255) / 256, (unsigned)num_sms() * 2), 256, 0, s, p);
  if (!p.general) launch_behind(k_table_halo, p.runs, TB_THREADS, sizeof(Tile), s, p);
}

void step_table(PipeDev &p, cudaStream_t s) {
  for (uint32_t part = 0; part < p.slices; part++) {
    const uint32_t n = (uint32_t)((unsigned long long)p.runs * (part + 1) / p.slices -
                                  (unsigned long long)p.runs * part / p.slices);
    if (n) launch_behind(k_table, n, TB_THREADS, sizeof(Tile), s, p, part, p.slices);
  }
}

}  // namespace stc
