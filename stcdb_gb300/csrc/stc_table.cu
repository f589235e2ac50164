// Step kernel (c), tiled: the table update, the ordered insertion of new
// meetings and the expire/emit sweep in one pass over the meeting table.
// Before and after, one GB300, per step: 10M uniform objects (2^28 slots,
// 67.7M hits, 36.7M of them new) 8.4 ms of pair tests with the update beside
// them and 2.7 of sweep -> 2.85 ms of pair tests and 2.9 of k_table (14.1 GB,
// 4.9 TB/s, 72% of the measured copy rate); hotspot-1M (34.7M hits) 4.0 + 1.9
// -> 1.7 + 2.3 ms (its blocks wait for their tiles: bound by HBM).
//
// The pair tests leave the step's hits binned by table tile (TILE_SLOTS
// slots, about; stc_refine.cu). A block takes a run of consecutive tiles and,
// tile by tile, copies the tile to shared memory, applies the tile's hits to
// it there (extensions, and claims of empty slots by priority), then
// finalises claims, clears or emits ended meetings and writes back the slots
// that changed. Applying the hits one by one at random over the table and
// sweeping it afterwards brought a 128-byte line from DRAM for every hit and
// the whole table again for the sweep; this way the table streams through
// once.
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
// takes the general path: k_hits, k_insert_ordered and k_sweep.
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

constexpr uint32_t TB_THREADS = 256;
constexpr uint32_t TB_BLOCKS_PER_SM = 5;
constexpr uint32_t TB_WAVES = 8;        // runs are short, so that query batches get SMs between them
constexpr uint32_t TB_RUN_TILES = 16;   // shortest run worth its halo, where the table has that many tiles
constexpr uint32_t TB_RECS = 256;       // hit records held in shared memory; the rest are read from the bin
constexpr uint32_t TB_STAGE = 48;       // emitted meetings staged per block
constexpr uint32_t TB_DUPS = 64;        // hits of possible double pairs listed per tile

// 44 KB, five blocks an SM: while one applies hits, the others' tiles load.
// (1024 slots and four blocks: 3.01 against 2.90 ms at 10M objects; 768 slots
// leave a tile's hits within one round of the block at a quarter's load.)
struct __align__(128) Tile {
  Slot slot[TILE_SLOTS];
  HitRec rec[TB_RECS];                  // the tile's hits, then those carried in
  uint32_t carry[2][TILE_LOAD];         // hits carried in and out: places counted from the run's first bin
  stc_meeting stage[TB_STAGE];
  uint32_t fresh[2 * TILE_LOAD];        // hits without a meeting: number | first empty slot << 16
  uint32_t dup[TB_DUPS];                // the same of possibly double ones
  unsigned long long bar;               // mbarrier of the tile's copies
  unsigned long long base;              // emit position of a staged batch
  // counters in turns, so that one is reset while its neighbours are in use
  uint32_t ncarry[3], ndup[2], nnew[2], live[2], nstage;
};

__device__ __forceinline__ unsigned long long tile_start(const PipeDev &p, uint32_t j) {
  const unsigned long long x = (unsigned long long)j * p.B;
  unsigned long long q = __umul64hi(x, p.nb_magic);  // x / nb: exact or one too large
  if (q * p.nb > x) q--;
  return q;
}

// Record `id` of a run whose bins are counted from tile r0 (cyclic).
__device__ __forceinline__ const HitRec *run_record(const PipeDev &p, uint32_t r0, uint32_t id) {
  const uint32_t seq = id / p.bin_cap;
  uint32_t tile = r0 + seq;
  if (tile >= p.nb) tile -= p.nb;
  return p.hits + (unsigned long long)tile * p.bin_cap + (id - seq * p.bin_cap);
}

__device__ __forceinline__ HitRec load_record(const HitRec *r) {
  const ulonglong2 v = *(const ulonglong2 *)r;
  const float4 m = *(const float4 *)&r->lo_x;
  HitRec h;
  h.a = (uint32_t)v.x;
  h.b = (uint32_t)(v.x >> 32);
  h.order = v.y;
  h.lo_x = m.x;
  h.lo_y = m.y;
  h.hi_x = m.z;
  h.hi_y = m.w;
  return h;
}

// ---- bulk copies into the tile, counted by an mbarrier ----

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(unsigned long long *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void bar_expect(unsigned long long *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_in(void *dst, const void *src, uint32_t bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// Waits for phase `parity` of the barrier; gives up after a bounded number
// of tries (false).
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, uint32_t parity) {
  for (uint32_t i = 0; i < (1u << 22); i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Starts the copies of tile `tile` and of its n hits (one thread).
__device__ __forceinline__ void tile_fetch(const PipeDev &p, Tile &s, uint32_t tile, unsigned long long start,
                                           uint32_t len, uint32_t n) {
  const uint32_t held = min(n, TB_RECS);
  // the block's earlier accesses to the buffers, ordered by its barrier,
  // come before the copies' writes
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  bar_expect(&s.bar, (len + held) * 32u);
  bulk_in(s.slot, p.slots + start, len * 32u, &s.bar);
  if (held) bulk_in(s.rec, p.hits + (unsigned long long)tile * p.bin_cap, held * 32u, &s.bar);
}

__device__ __forceinline__ uint32_t bin_hits(const PipeDev &p, uint32_t tile) {
  return min(p.bin_cnt[tile], p.bin_cap);
}

// The tile being worked on, as every thread sees it.
struct TileView {
  const HitRec *bin;         // the tile's bin
  unsigned long long start;  // its first slot
  uint32_t n, nc;            // its hits, hits carried in
  uint32_t r0, id0;          // the run's first bin, the place of this bin's first hit
  uint32_t len, turn;        // slots, the tile's number in its run
};

// Hit i of the tile (i < n: its own, then the ones carried in).
__device__ __forceinline__ const HitRec *tile_rec(const PipeDev &p, const Tile &s, const TileView &v, uint32_t i) {
  if (i < TB_RECS) return &s.rec[i];
  return i < v.n ? v.bin + i : run_record(p, v.r0, s.carry[v.turn & 1u][i - v.n]);
}

// First slot at or behind `pos` that holds `key` or is empty; v.len if none.
__device__ __forceinline__ uint32_t tile_probe(const Tile &s, const TileView &v, unsigned long long key, uint32_t pos,
                                               bool &found) {
  unsigned long long k = STC_EMPTY_KEY;
  for (; pos < v.len; pos++) {
    k = s.slot[pos].key;  // keys do not change while hits are applied
    if (k == key || k == STC_EMPTY_KEY) break;
  }
  found = pos < v.len && k == key;
  return pos;
}

// Hit i extends the meeting in its slot (tracing/refinement.cpp:40-42, MBR
// cuda/geometry.cu:474-478).
__device__ __forceinline__ void tile_extend(const PipeDev &p, Tile &s, const TileView &v, uint32_t i, uint32_t pos,
                                            uint32_t t) {
  const float4 m = *(const float4 *)&tile_rec(p, s, v, i)->lo_x;
  float4 *d = (float4 *)&s.slot[pos].lo_x;
  const float4 o = *d;
  s.slot[pos].end = t;
  *d = make_float4(fminf(o.x, m.x), fminf(o.y, m.y), fmaxf(o.z, m.z), fmaxf(o.w, m.w));
}

// Hit i, which found no meeting before slot `pos` (empty, or the tile's
// end): claims an empty slot, carrying on whatever it evicts; ends at a
// meeting of its own behind an empty slot it lost; or leaves the tile.
__device__ __forceinline__ void tile_claim(const PipeDev &p, Tile &s, const TileView &v, uint32_t i, uint32_t pos,
                                           uint32_t t) {
  const HitRec *h = tile_rec(p, s, v, i);
  unsigned long long key = stc_cantor(h->a, h->b), prio = h->order & ~DUP_BIT;
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
    if (found) {
      tile_extend(p, s, v, i, pos, t);
      return;
    }
    uint32_t *w = &s.slot[pos].start;
    uint32_t cur = atomicCAS(w, STC_NONE, i);
    if (cur == STC_NONE) return;  // settled: a new meeting
    for (;;) {  // a claimed slot stays claimed
      const HitRec *o = tile_rec(p, s, v, cur);
      const unsigned long long other = o->order & ~DUP_BIT;
      if (prio > other) break;  // lost this slot
      const uint32_t old = atomicCAS(w, cur, i);
      if (old == cur) {  // carry the evicted hit onward
        i = cur;
        key = stc_cantor(o->a, o->b);
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
// extended its meeting, claimed an empty slot (its start word names the hit)
// or been put on the other carry list. First every hit looks its meeting up,
// then the ones without one, packed together, claim slots: the two loops
// diverge little, where one loop for both had every warp wait for its longest
// chain of claims (8000 of 14600 cycles a tile at 10M objects; 7400 of 13300
// in two loops). Ends with the block's barrier.
__device__ __forceinline__ void tile_apply(const PipeDev &p, Tile &s, const TileView &v, uint32_t t) {
  const uint32_t tid = threadIdx.x, lt_mask = (1u << lane_id()) - 1u, par = v.turn & 1u;
  for (uint32_t i = tid; i < v.nc; i += TB_THREADS)
    if (v.n + i < TB_RECS) s.rec[v.n + i] = load_record(run_record(p, v.r0, s.carry[par][i]));
  if (!bar_wait(&s.bar, par)) stc_set_error(p.st, ERR_DA, (uint32_t)v.start);
  if (v.nc) __syncthreads();  // the carried records
  const uint32_t total = v.n + v.nc;
  for (uint32_t i0 = 0; i0 < total; i0 += TB_THREADS) {
    const uint32_t i = i0 + tid;
    bool claims = false;
    uint32_t pos = 0;
    if (i < total) {
      const HitRec *h = tile_rec(p, s, v, i);
      const unsigned long long key = stc_cantor(h->a, h->b);
      if (i < v.n) pos = (uint32_t)(fast_mod(key, p.B, p.B_magic) - v.start);
      bool found;
      pos = tile_probe(s, v, key, pos, found);
      if (found) {
        tile_extend(p, s, v, i, pos, t);
      } else if (i < v.n && (h->order & DUP_BIT)) {  // the pair's other instance decides which one claims
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
  for (uint32_t x = tid; x < m; x += TB_THREADS) tile_claim(p, s, v, s.fresh[x] & 0xFFFFu, s.fresh[x] >> 16, t);
  // hits flagged as possibly double: a pair's instances are in one bin, and
  // the one of lowest priority claims for all
  const uint32_t nd = s.ndup[par];
  if (nd) {
    const bool listed = nd <= TB_DUPS;
    for (uint32_t x = tid; x < (listed ? nd : v.n); x += TB_THREADS) {
      const uint32_t i = listed ? s.dup[x] & 0xFFFFu : x;
      const HitRec *h = tile_rec(p, s, v, i);
      const uint32_t a = h->a, b = h->b;
      const unsigned long long order = h->order;
      if (!(order & DUP_BIT)) continue;
      bool first = true;
      for (uint32_t y = 0; y < (listed ? nd : v.n) && first; y++) {
        const HitRec *o = tile_rec(p, s, v, listed ? s.dup[y] & 0xFFFFu : y);
        if (o->a == a && o->b == b && (o->order & DUP_BIT) && o->order < order) first = false;
      }
      if (!first) continue;
      uint32_t pos = s.dup[x & (TB_DUPS - 1)] >> 16;
      if (!listed) {
        const unsigned long long key = stc_cantor(a, b);
        bool found;
        pos = tile_probe(s, v, key, (uint32_t)(fast_mod(key, p.B, p.B_magic) - v.start), found);
        if (found) continue;  // extended already
      }
      tile_claim(p, s, v, i, pos, t);
    }
  }
  __syncthreads();
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

}  // namespace

// The largest bin and the largest (occupied slots + hits) of a tile, which
// decide the step's path (fuse_halo).
__global__ void __launch_bounds__(256) k_table_plan(PipeDev p) {
  uint32_t load = 0, most = 0;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < p.nb; j += gridDim.x * blockDim.x) {
    const uint32_t c = p.bin_cnt[j];
    most = max(most, c);
    load = max(load, c + p.tile_live[j]);
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
  extern __shared__ __align__(128) unsigned char smem[];
  Tile &s = *(Tile *)smem;
  const uint32_t halo = fuse_halo(p);
  if (!halo) return;
  const uint32_t t = p.st->step_t, tid = threadIdx.x;
  const uint32_t r = blockIdx.x;
  const uint32_t first = run_start(p, r), r0 = first >= halo ? first - halo : first + p.nb - halo;
  TileView v;
  v.r0 = r0;
  if (tid == 0) {
    bar_init(&s.bar);
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
    v.bin = p.hits + (unsigned long long)tile * p.bin_cap;
    if (tid == 0) tile_fetch(p, s, tile, v.start, v.len, v.n);
    tile_apply(p, s, v, t);
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
  extern __shared__ __align__(128) unsigned char smem[];
  Tile &s = *(Tile *)smem;
  const uint32_t halo = fuse_halo(p);
  if (!halo) return;
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
  if (tid == 0) {
    bar_init(&s.bar);
    s.ncarry[0] = nc;
    s.ncarry[1] = s.ncarry[2] = s.ndup[0] = s.ndup[1] = s.nnew[0] = s.nnew[1] = 0;
    s.live[0] = s.live[1] = s.nstage = 0;
    tile_fetch(p, s, first, v.start, v.len, v.n);
  }
  __syncthreads();
  for (uint32_t tile = first; tile < last; tile++) {
    v.turn = tile - first;
    v.id0 = (halo + v.turn) * p.bin_cap;
    v.bin = p.hits + (unsigned long long)tile * p.bin_cap;
    v.nc = min(s.ncarry[v.turn % 3], TILE_LOAD);
    const uint32_t next_n = tile + 1 < last ? bin_hits(p, tile + 1) : 0u;  // on its way beside the hits
    tile_apply(p, s, v, t);
    // write back what changed; clear and emit what ended (tracing/meeting.cpp:47-67)
    uint32_t live = 0;
    ulonglong2 ks[TILE_SLOTS / TB_THREADS];
#pragma unroll
    for (uint32_t u = 0; u < TILE_SLOTS / TB_THREADS; u++) {
      ks[u] = make_ulonglong2(STC_EMPTY_KEY, ~0ull);
      if (u * TB_THREADS + tid < v.len) ks[u] = *(const ulonglong2 *)&s.slot[u * TB_THREADS + tid];
    }
#pragma unroll
    for (uint32_t u = 0; u < TILE_SLOTS / TB_THREADS; u++) {
      const uint32_t i = u * TB_THREADS + tid;
      const ulonglong2 k = ks[u];
      bool emit = false;
      const uint32_t st = (uint32_t)k.y;
      float4 m = make_float4(STC_INIT_LO, STC_INIT_LO, STC_INIT_HI, STC_INIT_HI);
      if (k.x != STC_EMPTY_KEY || st != STC_NONE) {
        uint32_t start = STC_NONE, end = STC_NONE;
        unsigned long long key = STC_EMPTY_KEY;
        if (k.x == STC_EMPTY_KEY) {
          // a claim becomes a new meeting (cuda/geometry.cu:480-489): start =
          // end = t, MBR = init, then both objects' positions
          const HitRec *h = tile_rec(p, s, v, st);
          key = stc_cantor(h->a, h->b);
          start = end = t;
          m = make_float4(fminf(m.x, h->lo_x), fminf(m.y, h->lo_y), fmaxf(m.z, h->hi_x), fmaxf(m.w, h->hi_y));
          live++;
          fresh++;
        } else if ((uint32_t)(k.y >> 32) == t) {  // extended this step
          key = k.x;
          start = st;
          end = t;
          m = *(const float4 *)&s.slot[i].lo_x;
          live++;
        } else if (t - st >= p.min_meet_time + 1) {
          const float4 e = *(const float4 *)&s.slot[i].lo_x;
          emit = !p.mbr_filter ||
                 (e.x >= p.fmap_lo_x && e.z <= p.fmap_hi_x && e.y >= p.fmap_lo_y && e.w <= p.fmap_hi_y);
        }
        store_slot(&p.slots[v.start + i], key, start, end, m);
      }
      const uint32_t ball = __ballot_sync(0xffffffffu, emit);
      if (ball) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(&s.nstage, (uint32_t)__popc(ball));
        b = __shfl_sync(0xffffffffu, b, 0) + __popc(ball & lt_mask);
        if (emit) {
          stc_meeting e;
          cantor_decode(k.x, &e.pid_lo, &e.pid_hi);
          e.start = st;
          e.end = (uint32_t)(k.y >> 32);
          e.mbr[0] = s.slot[i].lo_x; e.mbr[1] = s.slot[i].lo_y; e.mbr[2] = s.slot[i].hi_x; e.mbr[3] = s.slot[i].hi_y;
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
    active += live;
    live = __reduce_add_sync(0xffffffffu, live);
    if (lane == 0 && live) atomicAdd(&s.live[v.turn & 1u], live);
    if (tid == 0) {
      const uint32_t next = (v.turn & 1u) ^ 1u;
      s.ncarry[(v.turn + 2) % 3] = s.ndup[next] = s.nnew[next] = s.live[next] = 0;
    }
    __syncthreads();
    const uint32_t staged = min(s.nstage, TB_STAGE);
    const bool flush = staged && (staged > TB_STAGE / 2 || tile + 1 == last);
    v.start += v.len;
    v.len = (uint32_t)(tile_start(p, min(tile + 2, p.nb)) - v.start);
    v.n = next_n;
    if (tid == 0) {
      if (tile + 1 < last) tile_fetch(p, s, tile + 1, v.start, v.len, next_n);
      p.tile_live[tile] = s.live[v.turn & 1u];
      if (flush) s.base = atomicAdd(&p.st->emit_count, (unsigned long long)staged);
    }
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

// Occupied slots of every tile, counted from the table (after a restore).
__global__ void k_tile_count(PipeDev p) {
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.B;
       i += (unsigned long long)gridDim.x * blockDim.x)
    if (p.slots[i].key != STC_EMPTY_KEY) atomicAdd(&p.tile_live[tile_of(p, i)], 1u);
}

static_assert(sizeof(Tile) + 1024 <= 228 * 1024 / TB_BLOCKS_PER_SM, "blocks per SM");

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
  p.runs = std::min(p.nb, std::min(wave * TB_WAVES, std::max(wave, p.nb / TB_RUN_TILES)));
}

void count_tiles(PipeDev &p, cudaStream_t s) {
  cudaMemsetAsync(p.tile_live, 0, (size_t)p.nb * sizeof(uint32_t), s);
  STC_KL k_tile_count<<<num_sms() * 8, 256, 0, s>>>(p);
}

void step_table_plan(PipeDev &p, cudaStream_t s) {
  STC_KL k_table_plan<<<std::min<unsigned>((p.nb + 255) / 256, (unsigned)num_sms() * 2), 256, 0, s>>>(p);
  STC_KL k_table_halo<<<p.runs, TB_THREADS, sizeof(Tile), s>>>(p);
}

void step_table(PipeDev &p, cudaStream_t s) {
  for (uint32_t part = 0; part < p.slices; part++) {
    const uint32_t n = (uint32_t)((unsigned long long)p.runs * (part + 1) / p.slices -
                                  (unsigned long long)p.runs * part / p.slices);
    if (n) STC_KL k_table<<<n, TB_THREADS, sizeof(Tile), s>>>(p, part, p.slices);
  }
}

}  // namespace stc
