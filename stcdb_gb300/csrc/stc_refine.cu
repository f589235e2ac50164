// Step kernel (b): proximity refinement, and the general path's table update.
//
// Work: every leaf's n kept members (the first leaf_cap in pid order,
// tracing/filter.cpp:100-104) are ordered by horizontal strips at least
// reach tall and, within small strips, by longitude (stc_partition.cu,
// k_leaf_small). The reference tests every own-leaf pair (pid < q,
// tracing/refinement.cpp:30) and every (border unit, member) pair of the
// leaf (tracing/filter.cpp:248-259); a pair more than a strip apart, or
// farther apart in longitude than the leaf's window wx, is farther than
// reach, so only the pairs in a member's candidate windows -- the members
// after it in its strip up to its window's end and its window in the next
// strip, or for a border unit its window in the three strips beside its
// point -- can hit, and only those are tested. A job is 32 rows (members or
// border units) of one leaf, one per lane, each over one chunk of
// refine_chunk positions of its own contiguous segments (a dense leaf's
// n^2 / 2 pair tests spread over many jobs). Each hit keeps the reference's
// priority: the finding unit's rank, then the member's pid, which orders a
// leaf's members as their place in the reference's pid-ordered list does.
//
// Distance decisions equal the reference's fp64 test
// `p1->distance(p2, true) <= reach` (tracing/refinement.cpp:30-33,
// geometry/geometry.h:40-48). Each pair is first classified in fp32 from the
// points' offsets to the leaf corner; the classification is conservative by
// construction (error bound below), and only pairs inside the uncertainty
// band are recomputed with the reference's exact fp64 expression.
//
// Error bound of the fp32 estimate d_f of the reference distance d, with
// u = 2^-24, X = |x - corner| <= mx (degrees lon), Y <= my (degrees lat):
//   offsets round with |err| <= u X, so dx picks up <= 2 u mx degrees and dy
//   <= 2 u my; the rest (subtraction, scale factor from sinf, products, sum)
//   is relative and below 30 u. Hence
//     |d_f - d| <= 30 u d + 2.1 u (2 mx SMAX + 2 my SLAT) = 30 u d + E.
//   A pair is accepted when d_f^2 <= (r - delta)^2 and rejected when
//   d_f^2 >= (r + delta)^2 with delta = 4E + 64 u r + 1e-6 r, which leaves
//   slack for the rounding of the squared thresholds themselves.
//
// Hits (tracing/refinement.cpp:34-55) go to the bin of the table tile their
// home slot key % B lies in, with their position in the reference's
// sequential processing order: unit rank << order_shift | pid. stc_table.cu
// applies them; the general path here does so for a step whose tiles are too
// full (k_hits) and for the steps told so beforehand, whose hits are not binned
// (k_hits_part): a key found before the first empty slot is extended in place
// (end = t, MBR), every other key walks on for a slot by priority.
#include <algorithm>

#include "stc_insert.cuh"

namespace stc {


__device__ __forceinline__ double dpml_fast_r(double lat) {
  double absla = fabs(lat);
  if (absla == 90) absla = 89;
  double arg = RN_DIV(RN_MUL(RN_SUB(90.0, absla), STC_REF_PI), 180.0);
  return RN_DIV(360.0, RN_MUL(RN_MUL(sin(arg), 40076.0), 1000.0));
}

// Reference distance decision for p1 (whose latitude sets the scale) and p2.
// (not inlined: about 1 in 180,000 tests comes here)
__device__ __noinline__ bool exact_within(const PipeDev &p, uint32_t pid1, uint32_t pid2, uint32_t &amb) {
  double2 a = p.xy[pid1], b = p.xy[pid2];
  double d = stc_distance_ref(a.x, a.y, b.x, b.y, dpml_fast_r(a.y));
  if (fabs(d - p.reach) > 1e-12 * p.reach) return d <= p.reach;
  d = stc_distance_ref(a.x, a.y, b.x, b.y, stc_dpml_ref(a.y));
  // within a few ulp of reach the decision depends on the last bit of sin()
  if (fabs(d - p.reach) <= 8.0 * 2.220446049250313e-16 * p.reach) amb++;
  return d <= p.reach;
}

// Merges one instance of a key that may occur twice in this step into the
// candidate set (minimum priority); the candidate pass walks it afterwards.
__device__ void cand_insert(const PipeDev &p, unsigned long long key, unsigned long long order) {
  unsigned long long h = mix64(key) & (p.C - 1);
  for (unsigned long long probe = 0; probe < STC_PROBE_LIMIT; probe++) {
    Cand *c = &p.cset[h];
    unsigned long long k = *(volatile unsigned long long *)&c->key;
    if (k == STC_EMPTY_KEY) {
      // the list bounds the set's load factor at cand_cap / C <= 1/2
      if (*(volatile unsigned long long *)&p.st->cand_count >= p.cand_cap) {
        stc_set_error(p.st, ERR_CAND, 0u);
        return;
      }
      k = atomicCAS(&c->key, STC_EMPTY_KEY, key);
      if (k == STC_EMPTY_KEY) {
        unsigned long long n = agg_inc(&p.st->cand_count);
        if (n < p.cand_cap) p.cand_list[n] = (uint32_t)h;
        else stc_set_error(p.st, ERR_CAND, (uint32_t)n);
        k = key;
      }
    }
    if (k == key) {
      atomicMin(&c->order, order);
      return;
    }
    h = (h + 1) & (p.C - 1);
  }
  stc_set_error(p.st, ERR_CAND, 0xFFFFFFFFu);
}


// Applies one hit (key = cantor(h.a, h.b)) to the table. kv/mbr: the slot
// at key % B, already loaded.
__device__ void process_hit_at(const PipeDev &p, const HitRec &h, unsigned long long key, uint32_t t,
                               unsigned long long slot, U128 kv, float4 mbr) {
  for (unsigned long long probe = 0; probe < STC_PROBE_LIMIT && probe < p.B; probe++) {
    Slot *s = &p.slots[slot];
    if (kv.lo == key) {  // tracing/refinement.cpp:40-42 (+ MBR, cuda/geometry.cu:474-478)
      s->end = t;
      // the box of both objects' float positions this step comes with the
      // record; the MBR only grows during a step, so a stale read of it can
      // only cause an extra atomic
      if (h.lo_x < mbr.x) atomic_min_f(&s->lo_x, h.lo_x);
      if (h.lo_y < mbr.y) atomic_min_f(&s->lo_y, h.lo_y);
      if (h.hi_x > mbr.z) atomic_max_f(&s->hi_x, h.hi_x);
      if (h.hi_y > mbr.w) atomic_max_f(&s->hi_y, h.hi_y);
      return;
    }
    if (kv.lo == STC_EMPTY_KEY || (kv.lo & STC_CLAIM_BIT)) {  // empty before this step: a new key
      if (h.order & DUP_BIT) {
        cand_insert(p, key, h.order & ~DUP_BIT);
      } else {
        if (!ordered_walk(p, key, h.order, slot, t, &kv)) stc_set_error(p.st, ERR_DA, (uint32_t)slot);
      }
      return;
    }
    slot = slot + 1 == p.B ? 0 : slot + 1;
    kv = load_slot_pair(&p.slots[slot]);
    mbr = __ldcg((const float4 *)&p.slots[slot].lo_x);
  }
  stc_set_error(p.st, ERR_PROBE, (uint32_t)slot);
}

// (not inlined: it would cost the pair tests' loop its registers)
__device__ __noinline__ void process_hit(const PipeDev &p, const HitRec &h, uint32_t t) {
  const unsigned long long key = stc_cantor(h.a, h.b);
  unsigned long long slot = fast_mod(key, p.B, p.B_magic);
  process_hit_at(p, h, key, t, slot, load_slot_pair(&p.slots[slot]), __ldcg((const float4 *)&p.slots[slot].lo_x));
}

// One 32-byte store: a whole sector per record (a plain assignment is split
// into narrower stores, each a partial write of the sector in L2: 10M uniform
// objects, 67.7M records a step, pair tests 5.8 ms with it).
__device__ __forceinline__ void store_hit(HitRec *d, const HitRec &h) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(d), "r"(h.a), "r"(h.b),
               "r"((uint32_t)h.order), "r"((uint32_t)(h.order >> 32)), "r"(__float_as_uint(h.lo_x)),
               "r"(__float_as_uint(h.lo_y)), "r"(__float_as_uint(h.hi_x)), "r"(__float_as_uint(h.hi_y))
               : "memory");
}

// Appends one hit to the bin of the table tile its home slot lies in, where
// the table update finds the tile's hits together. The records are 32-byte
// sectors whose bins' open ends stay in L2 (one 128-byte line a bin: 45 MB
// for 2^28 slots), so they reach HBM as whole lines. A hit its bin has no
// room for is applied here, and the step then takes the general path; while
// the tiles are packed that has to wait until they are unpacked, and the pair
// tests are done once more (k_hits).
__device__ __forceinline__ void bin_hit(const PipeDev &p, const HitRec &h, uint32_t t) {
  const unsigned long long key = stc_cantor(h.a, h.b);
  const uint32_t bin = tile_of(p, fast_mod(key, p.B, p.B_magic));
  const uint32_t pos = atomicAdd(&p.bin_cnt[bin], 1u);
  if (pos < p.bin_cap) store_hit(&p.hits[hit_place(p, bin, pos)], h);
  else if (p.st->packed == TABLE_SLOTS) process_hit(p, h, t);
  else p.st->redo = 1;
}

// Steps told to be general (PathChoice) leave their hits in sequence instead: a
// warp takes HIT_WINDOW places of the buffer at a time, more the more it has
// taken (508M hits in windows of 64, 256, up to 1024: 102, 94, 94 ms a step, by
// the shared counter), and the rest of its last ones stay empty (a = STC_NONE).
// Random to the table, but the update of one part runs beside the tests of the
// next, and a crowd's long walks are spread over all warps (figures at
// PathChoice).
constexpr uint32_t HIT_WINDOW = 64, HIT_WINDOW_MOST = 1024;
struct HitWindow {
  unsigned long long next, end;  // the same for the whole warp
  uint32_t taken;                // places so far
};
__device__ __forceinline__ void window_rest(const PipeDev &p, const HitWindow &w) {
  const unsigned long long room = hit_records(p.nb, p.bin_cap);
  for (unsigned long long i = w.next + lane_id(); i < w.end; i += 32)
    if (i < room) p.hits[i].a = STC_NONE;
}
// The round's hits (one a lane with has set); the ones the buffer has no room
// for are applied here. Called by the whole warp.
__device__ __forceinline__ void append_round(const PipeDev &p, const HitRec &h, bool has, uint32_t t, HitWindow &w) {
  const uint32_t hm = __ballot_sync(0xffffffffu, has), cnt = __popc(hm);
  if (w.end - w.next < cnt) {
    window_rest(p, w);
    const uint32_t size = min(max(w.taken / 4, HIT_WINDOW), HIT_WINDOW_MOST);
    unsigned long long base = 0;
    if (lane_id() == 0) base = atomicAdd(&p.st->hit_count, (unsigned long long)size);
    w.next = __shfl_sync(0xffffffffu, base, 0);
    w.end = w.next + size;
    w.taken += size;
  }
  if (has) {
    const unsigned long long pos = w.next + __popc(hm & ((1u << lane_id()) - 1u));
    if (pos < hit_records(p.nb, p.bin_cap)) store_hit(&p.hits[pos], h);
    else process_hit(p, h, t);
  }
  w.next += cnt;
}

__device__ __forceinline__ HitRec load_hit(const HitRec *r) {
  // streamed once: evict-first loads keep L2 for the table and positions
  const ulonglong2 v = __ldcs((const ulonglong2 *)r);
  const float4 m = __ldcs((const float4 *)&r->lo_x);
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

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct Counters {
  uint32_t tests, exact, hits, amb;  // per thread; summed into 64-bit totals per warp
};

// First index in [lo, hi) of a longitude-ordered strip whose offset is
// greater than x (upper) or not below x (!upper).
__device__ __forceinline__ uint32_t strip_x_bound(const float4 *pts, uint32_t lo, uint32_t hi, float x, bool upper) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    const float v = __ldg(&pts[mid]).x;
    if (upper ? v <= x : v < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// One row (an own member or a border unit) of the job a warp works on, in
// shared memory: its point, its candidate segments and where its tests start
// among the job's. 80 bytes apart, so that 16-byte reads of different rows
// fall in different banks.
struct __align__(16) Row {
  float x, y, scale;         // leaf offsets, metres per degree of longitude
  uint32_t pid;
  float fx, fy;              // float position
  uint32_t off;              // first test of the row among the job's
  uint32_t unit;             // border: place of the unit
  uint32_t seg0, seg1, seg2; // segments: start | end (counted in the row's tests) << 16; start only in seg2
  uint32_t leaf;             // border: the leaf of the row's point, and its low x, low y, high y in float
  float ax0, ay0, ay1;
  uint32_t pad[5];
};

// One job: 32 rows of leaf g, each against its candidate ranges of members
// in (strip, longitude) order (stc_partition.cu, k_leaf_small). Rows are
// the leaf's own members (own = true; row i tests the members after it in
// its strip up to its longitude window's end, and its window in the next
// strip, so every pair of members within reach is tested once) or 32 border
// units targeting the leaf (the members in the unit's longitude window in
// the three strips beside its point). A row's candidates come in up to
// three contiguous segments, of which the job takes one chunk of refine_chunk
// positions. The job's tests are numbered through, row after row, and each
// lane takes every 32nd, hit or miss: rows have 8 candidates on average but
// the longest of 32 has several times that, and with a row per lane 17 of 32
// lanes had work. The tests alone, without records: 1.15 ms of a 10M-object
// step (93.6M tests, 67.7M hits); with the bins' counters 1.55, with the
// records' stores 2.85, or 2.4 in chunks (hit_place): bound by the rate of
// scattered stores over that many pages (52 G/s measured). A row per lane and a shared-memory queue
// of records before it: 3.0 ms for the tests with sequential records.
// HITS_APPLY: every hit is applied to the table at once, nothing is binned; the
// schema is not read, which its update may be rewriting.
enum HitsGo { HITS_BIN, HITS_APPLY, HITS_APPEND };
template <HitsGo GO>
__device__ void run_rows(const PipeDev &p, uint32_t g, bool own, uint32_t rowblock, uint32_t chunk, uint32_t t,
                         Counters &ct, Row *rows, HitWindow &window) {
  constexpr bool REDO = GO == HITS_APPLY;
  const uint32_t lane = lane_id();
  const LeafGeo *lg = &p.lgeo[g];
  const uint32_t base = lg->base, n = lg->n;
  const float ext_x = lg->ext_x, ext_y = lg->ext_y;
  float x = 0.f, y = 0.f, scale = 0.f, ax0 = 0.f, ay0 = 0.f, ay1 = 0.f;
  float2 fr = make_float2(0.f, 0.f);
  uint32_t pid = 0, unit = 0, leaf = 0;
  uint32_t sa0 = 0, sa1 = 0, sa2 = 0, sl0 = 0, sl1 = 0, sl2 = 0;  // candidate segments: start, length
  if (own) {
    const uint32_t i = rowblock * 32 + lane;
    if (i < n) {
      const float4 rp = __ldg(&p.spts[base + i]);
      fr = __ldg(&p.sfxy[base + i]);
      x = rp.x;
      y = rp.y;
      scale = rp.z;
      pid = __float_as_uint(rp.w);
      const uint2 c = __ldg(&p.scand[base + i]);
      const uint32_t e1 = c.x & 0xFFFFu, a2 = c.x >> 16;
      sa0 = i + 1;
      sl0 = e1 > i + 1 ? e1 - (i + 1) : 0u;
      sa1 = a2;
      sl1 = c.y > a2 ? c.y - a2 : 0u;
    }
  } else {
    const uint32_t i = rowblock * 32 + lane;
    if (i < p.bu_cnt[g]) {
      unit = p.bu_sorted_pos[p.bu_start[g] + i];
      pid = p.bu_pid[unit];
      const double2 qq = p.xy[pid];
      fr = float_pos(qq);
      x = __double2float_rn(RN_SUB(qq.x, lg->lo_x));
      y = __double2float_rn(RN_SUB(qq.y, lg->lo_y));
      scale = metres_per_deg_lon_f(fr.y);
      // A pair of a border row (outside leaf g) and a member occurs twice in
      // this step iff the member also has a border unit targeting the row's
      // leaf.
      leaf = p.leaf_gid[pid];
      if (!REDO) {
        const Node *ro = &p.sd.nodes[p.sd.gid_node[leaf]];
        ax0 = __double2float_rn(ro->lo_x);
        ay0 = __double2float_rn(ro->lo_y);
        ay1 = __double2float_rn(ro->hi_y);
      }
      // candidates: the members in the point's longitude window of the
      // strips beside its own (all of a strip too large to be ordered)
      const int H = (int)lg->strips;
      const float wx = lg->wx;
      const int c = (int)fminf(fmaxf(floorf(y * lg->inv), -4.0f), (float)H + 4.0f);
      const uint16_t *ss = p.sstart + (size_t)g * STRIP_STRIDE;
      const float4 *sp = p.spts + base;
      auto candidates = [&](int sidx, uint32_t &a, uint32_t &len) {
        if (sidx < 0 || sidx >= H) return;
        const uint32_t st = ss[sidx], en = ss[sidx + 1];
        uint32_t lo = st, hi = en;
        if (en - st >= 2 && en - st <= XSORT_MAX) {
          lo = strip_x_bound(sp, st, en, x - wx, false);
          hi = strip_x_bound(sp, lo, en, x + wx, true);
        }
        a = lo;
        len = hi - lo;
      };
      candidates(c - 1, sa0, sl0);
      candidates(c, sa1, sl1);
      candidates(c + 1, sa2, sl2);
    }
  }
  // this job's chunk: positions [chunk * refine_chunk, (chunk + 1) *
  // refine_chunk) of the row's segments taken one after the other
  {
    uint32_t skip = chunk * p.refine_chunk, take = p.refine_chunk;
    auto cut = [&](uint32_t &a, uint32_t &len) {
      const uint32_t d = min(skip, len);
      a += d;
      skip -= d;
      len = min(take, len - d);
      take -= len;
    };
    cut(sa0, sl0);
    cut(sa1, sl1);
    cut(sa2, sl2);
  }
  // the rows that have tests, with the number of their first one
  const uint32_t len = sl0 + sl1 + sl2;
  uint32_t incl = len;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
    if ((int)lane >= d) incl += up;
  }
  const uint32_t off = incl - len, total = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t nz = __ballot_sync(0xffffffffu, len != 0);
  // error margin: offsets of the members are within the leaf's extent; a
  // border row's own offsets may exceed it
  const float wxl = ext_x * 1.000001f, wyl = ext_y * 1.000001f;
  const float mx = fmaxf(wxl, warp_max(fabsf(x))), my = fmaxf(wyl, warp_max(fabsf(y)));
  if (len) {
    float4 *d = (float4 *)&rows[__popc(nz & ((1u << lane) - 1u))];
    d[0] = make_float4(x, y, scale, __uint_as_float(pid));
    d[1] = make_float4(fr.x, fr.y, __uint_as_float(off), __uint_as_float(unit));
    *(uint4 *)&d[2] = make_uint4(sa0 | sl0 << 16, sa1 | (sl0 + sl1) << 16, sa2, leaf);
    if (!own) d[3] = make_float4(ax0, ay0, ay1, 0.f);
  }
  __syncwarp();
  const float u = 5.9604645e-08f;
  const float reach = p.reach_f;
  const float E = 2.1f * u * (2.0f * mx * STC_SMAX_F + 2.0f * my * STC_SLAT_F);
  const float delta = 4.0f * E + 64.0f * u * reach + 1e-6f * reach;
  const float lo = fmaxf(reach - delta, 0.0f);
  const float lo2 = lo * lo;
  const float hi2 = (reach + delta) * (reach + delta);
  uint32_t before = 0;  // rows that started before this round
  for (uint32_t f0 = 0; f0 < total; f0 += 32) {
    // one bit per test of the round that is its row's first
    const uint32_t starts = __reduce_or_sync(0xffffffffu, len != 0 && off - f0 < 32u ? 1u << (off - f0) : 0u);
    const uint32_t ri = before + __popc(starts & (0xffffffffu >> (31u - lane))) - 1u;
    before += __popc(starts);
    // this lane's test; its record if it is a hit
    auto test = [&](HitRec &h) {
      const Row *w = &rows[ri];
      const float4 rp = *(const float4 *)w;
      const float4 r1 = *((const float4 *)w + 1);
      const uint4 r2 = *((const uint4 *)w + 2);
      const uint32_t k = f0 + lane - __float_as_uint(r1.z);
      const uint32_t e0 = r2.x >> 16, e1 = r2.y >> 16;
      const uint32_t j = base + (k < e0 ? (r2.x & 0xFFFFu) + k : k < e1 ? (r2.y & 0xFFFFu) + k - e0 : r2.z + k - e1);
      const float4 c = __ldg(&p.spts[j]);
      const float2 fc = __ldg(&p.sfxy[j]);
      const uint32_t pid1 = __float_as_uint(rp.w), pid2 = __float_as_uint(c.w);
      const bool less = pid1 < pid2;
      // the reference measures from the unit's point: an own pair from its
      // lower pid (tracing/refinement.cpp:30), a border pair from the unit
      const bool swap = own && !less;
      const float dx = (rp.x - c.x) * (swap ? c.z : rp.z);
      const float dy = (rp.y - c.y) * STC_SLAT_F;
      const float d2 = dx * dx + dy * dy;
      ct.tests++;
      bool hit = d2 <= lo2;
      if (!hit && d2 < hi2) {
        ct.exact++;
        hit = swap ? exact_within(p, pid2, pid1, ct.amb) : exact_within(p, pid1, pid2, ct.amb);
      }
      if (!hit) return false;
      ct.hits++;
      h.a = less ? pid1 : pid2;
      h.b = less ? pid2 : pid1;
      const float2 f1 = make_float2(r1.x, r1.y), fa = less ? f1 : fc, fb = less ? fc : f1;
      h.lo_x = fminf(fa.x, fb.x);
      h.lo_y = fminf(fa.y, fb.y);
      h.hi_x = fmaxf(fa.x, fb.x);
      h.hi_y = fmaxf(fa.y, fb.y);
      if (own) {
        // the pair is found by the lower pid's own unit (rank = its pid) at
        // the higher pid's place in the pid-ordered member list
        h.order = ((unsigned long long)h.a << p.order_shift) | h.b;
      } else {
        // border units follow the N own units
        h.order = (((unsigned long long)p.N + __float_as_uint(r1.w)) << p.order_shift) | pid2;
        // the member has a unit targeting the row's leaf only if it lies below
        // that leaf, or left of it and below its top (the border lookup's
        // rule); rounding to float keeps the order, so the test on floats
        // passes every such member, and the three dependent loads of its units
        // are left to the few that pass
        const float4 r3 = *((const float4 *)w + 3);
        if (REDO || fc.y <= r3.y || (fc.y <= r3.z && fc.x <= r3.x)) {
          const uint32_t cnb = p.bcount[pid2];
          const uint32_t coff = cnb ? p.boff[pid2] : 0u;
          for (uint32_t u2 = 0; u2 < cnb; u2++)
            if (p.bu_gid[coff + u2] == r2.w) h.order |= DUP_BIT;
        }
      }
      return true;
    };
    HitRec h;
    if (GO == HITS_APPEND) {
      const bool has = f0 + lane < total && test(h);
      append_round(p, h, has, t, window);
    } else if (f0 + lane < total && test(h)) {
      if (REDO) process_hit(p, h, t);
      else bin_hit(p, h, t);
    }
  }
  __syncwarp();
}

// The pair tests of a step whose bins overflowed while the table's tiles were
// packed, once more: part `part` of `parts` of the jobs, by the whole grid.
__device__ __noinline__ void redo_pairs(const PipeDev &p, Row *rows, uint32_t part, uint32_t parts) {
  const uint32_t t = p.st->step_t;
  const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  const unsigned long long J = p.st->jobs_total, J1 = J * (part + 1) / parts;
  Counters ct = {0, 0, 0, 0};  // counted the first time
  HitWindow none = {0, 0, 0};
  for (unsigned long long job = J * part / parts + warp; job < J1; job += nwarps) {
    if (__shfl_sync(0xffffffffu, (int)stc_failed(p.st), 0)) break;
    const uint4 w = p.jobs[job];
    for (uint32_t c = 0; c < w.w; c++)
      run_rows<HITS_APPLY>(p, w.x, (w.y & JOB_OWN) != 0, w.y & ~JOB_OWN, w.z + c, t, ct, rows, none);
  }
}

// The general path's table update: each lane takes HITS_LANE hits of a bin of
// its own, two in flight (both records and both home slots are requested before
// either is used). Lanes of one bin meet in the same few lines with their
// claims, and more registers, for redo_pairs, leave fewer warps: 371M hits in a
// table of 2^30 slots, two thirds of its slots and hits a tile, 85 ms with a
// warp a bin and 80 registers, 63 this way.
// Part `part` of `parts` takes that part of the bins.
constexpr uint32_t HITS_LANE = 8;
__global__ void __launch_bounds__(256, 5) k_hits(PipeDev p, uint32_t part, uint32_t parts) {
  after_previous();
  if (fuse_halo(p)) return;
  __shared__ Row rows_all[256 / 32][32];
  if (p.st->redo) {
    redo_pairs(p, rows_all[threadIdx.x >> 5], part, parts);
    return;
  }
  const uint32_t t = p.st->step_t;
  const uint32_t turns = (min((uint32_t)p.st->hit_max, p.bin_cap) + HITS_LANE - 1) / HITS_LANE;  // of the fullest bin
  const uint32_t groups = (p.nb + 31u) / 32u;
  const uint32_t g0 = (uint32_t)((unsigned long long)groups * part / parts);
  // (a 256th of the records that the buffer has room for, about)
  const uint32_t total = ((uint32_t)((unsigned long long)groups * (part + 1) / parts) - g0) * turns;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total; w += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t bin = (g0 + w / turns) * 32u + lane_id(), i0 = w % turns * HITS_LANE;
    if (bin >= p.nb) continue;
    const uint32_t n = min(min(p.bin_cnt[bin], p.bin_cap), i0 + HITS_LANE);
    for (uint32_t i = i0; i < n; i += 2) {
      const bool two = i + 1 < n;
      const HitRec h0 = load_hit(&p.hits[hit_place(p, bin, i)]);
      const HitRec h1 = load_hit(&p.hits[hit_place(p, bin, two ? i + 1 : i)]);
      const unsigned long long k0 = stc_cantor(h0.a, h0.b), k1 = stc_cantor(h1.a, h1.b);
      const unsigned long long s0 = fast_mod(k0, p.B, p.B_magic), s1 = fast_mod(k1, p.B, p.B_magic);
      const U128 kv0 = load_slot_pair(&p.slots[s0]), kv1 = load_slot_pair(&p.slots[s1]);
      const float4 m0 = __ldcg((const float4 *)&p.slots[s0].lo_x), m1 = __ldcg((const float4 *)&p.slots[s1].lo_x);
      process_hit_at(p, h0, k0, t, s0, kv0, m0);
      if (two) process_hit_at(p, h1, k1, t, s1, kv1, m1);
    }
  }
}

// Slice `part` of `parts` runs jobs [J * part / parts, J * (part + 1) / parts),
// dealt out beforehand, up to p.job_chunk at a time; fewer when there are too
// few to go round: eight dense jobs of one leaf in one warp were the whole
// kernel's tail (20k objects in hotspots: 0.23 -> 0.06 ms a quarter). SHARE
// (job_share): a warp takes its next job from a common counter instead, and a
// quarter more than its share at most, so that blocks still end, and let query
// batches in, during the kernel.
// APPEND: the hits in sequence (append_round).
template <bool SHARE, bool APPEND>
__global__ void __launch_bounds__(REFINE_THREADS, 4) k_refine_a(PipeDev p, uint32_t part, uint32_t parts) {
  __shared__ Row rows_all[REFINE_THREADS / 32][32];
  Row *rows = rows_all[threadIdx.x >> 5];
  const uint32_t t = p.st->step_t;
  const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  const unsigned long long J = p.st->jobs_total;
  const unsigned long long J0 = J * part / parts, J1 = J * (part + 1) / parts;
  const unsigned long long each = (J1 - J0) / nwarps;
  const unsigned long long jc = SHARE || !each ? 1ull : each >= p.job_chunk ? p.job_chunk : each;
  const unsigned long long quota = each + each / 4 + 2;
  Counters ct = {0, 0, 0, 0};
  HitWindow window = {0, 0, 0};
  unsigned long long taken = 0;
  for (unsigned long long j0 = J0 + warp * jc; j0 < J1;) {
    // one lane reads the flag so that the whole warp leaves together
    if (__shfl_sync(0xffffffffu, (int)stc_failed(p.st), 0)) break;
    unsigned long long next = j0 + nwarps * jc;
    if (SHARE) {  // asked for ahead of the job at hand
      next = J1;
      if (++taken < quota && lane_id() == 0) next = J0 + nwarps + atomicAdd(&p.ctr[CTR_JOBS + part], 1ull);
    }
    const unsigned long long j1 = j0 + jc < J1 ? j0 + jc : J1;
    for (unsigned long long job = j0; job < j1; job++) {
      const uint4 w = p.jobs[job];
      for (uint32_t c = 0; c < w.w; c++)
        run_rows<APPEND ? HITS_APPEND : HITS_BIN>(p, w.x, (w.y & JOB_OWN) != 0, w.y & ~JOB_OWN, w.z + c, t, ct, rows,
                                                  window);
    }
    j0 = SHARE ? __shfl_sync(0xffffffffu, next, 0) : next;
  }
  if (APPEND) window_rest(p, window);
  // reduce counters per warp (64-bit sums)
  unsigned long long tests = ct.tests, exact = ct.exact, hits = ct.hits, amb = ct.amb;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tests += __shfl_xor_sync(0xffffffffu, tests, o);
    exact += __shfl_xor_sync(0xffffffffu, exact, o);
    hits += __shfl_xor_sync(0xffffffffu, hits, o);
    amb += __shfl_xor_sync(0xffffffffu, amb, o);
  }
  if (lane_id() == 0) {
    if (tests) atomicAdd(&p.st->tests, tests);
    if (exact) atomicAdd(&p.st->exact_tests, exact);
    if (hits) atomicAdd(&p.st->hits, hits);
    if (amb) atomicAdd(&p.st->ambiguous, amb);
  }
}

void step_pairs(PipeDev &p, cudaStream_t s) {
  for (uint32_t part = 0; part < p.slices; part++) {
    const unsigned blocks = num_sms() * refine_blocks(p);
    if (p.job_share) STC_KL k_refine_a<true, false><<<blocks, REFINE_THREADS, 0, s>>>(p, part, p.slices);
    else STC_KL k_refine_a<false, false><<<blocks, REFINE_THREADS, 0, s>>>(p, part, p.slices);
  }
}

// hit_bounds[part + 1] = the end of the hits after part `part` (parts run in
// stream order).
__global__ void k_hit_mark(PipeDev p, uint32_t part) {
  const unsigned long long n = p.st->hit_count, room = hit_records(p.nb, p.bin_cap);
  p.hit_bounds[part + 1] = n < room ? n : room;
  if (part == 0) p.hit_bounds[0] = 0;
}

// The table update of part `part`'s hits, one thread per hit, two in flight:
// both records and both home slots are requested before either is used.
__global__ void __launch_bounds__(256) k_hits_part(PipeDev p, uint32_t part) {
  const uint32_t t = p.st->step_t;
  const unsigned long long first = p.hit_bounds[part], end = p.hit_bounds[part + 1];
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = first + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < end;
       i += 2 * stride) {
    const HitRec h0 = load_hit(&p.hits[i]);
    HitRec h1;
    h1.a = STC_NONE;
    if (i + stride < end) h1 = load_hit(&p.hits[i + stride]);
    const bool v0 = h0.a != STC_NONE, v1 = h1.a != STC_NONE;
    const unsigned long long k0 = v0 ? stc_cantor(h0.a, h0.b) : 0, k1 = v1 ? stc_cantor(h1.a, h1.b) : 0;
    const unsigned long long s0 = fast_mod(k0, p.B, p.B_magic), s1 = fast_mod(k1, p.B, p.B_magic);
    U128 kv0 = {0, 0}, kv1 = {0, 0};
    float4 m0 = make_float4(0.f, 0.f, 0.f, 0.f), m1 = m0;
    if (v0) {
      kv0 = load_slot_pair(&p.slots[s0]);
      m0 = __ldcg((const float4 *)&p.slots[s0].lo_x);
    }
    if (v1) {
      kv1 = load_slot_pair(&p.slots[s1]);
      m1 = __ldcg((const float4 *)&p.slots[s1].lo_x);
    }
    if (v0) process_hit_at(p, h0, k0, t, s0, kv0, m0);
    if (v1) process_hit_at(p, h1, k1, t, s1, kv1, m1);
  }
}

void step_pairs_part(PipeDev &p, uint32_t part, uint32_t parts, cudaStream_t s) {
  const unsigned blocks = num_sms() * refine_blocks(p);
  if (p.job_share) STC_KL k_refine_a<true, true><<<blocks, REFINE_THREADS, 0, s>>>(p, part, parts);
  else STC_KL k_refine_a<false, true><<<blocks, REFINE_THREADS, 0, s>>>(p, part, parts);
  STC_KL k_hit_mark<<<1, 1, 0, s>>>(p, part);
}

// (twice the blocks of k_hits: few hits a thread, so that the pair tests' blocks
// find room beside them; 16, 32 blocks an SM: 94.2, 89.7 ms a step)
void step_hits_part(PipeDev &p, uint32_t part, cudaStream_t s) {
  STC_KL k_hits_part<<<num_sms() * 2 * p.hits_bps, 256, 0, s>>>(p, part);
}

void step_hits(PipeDev &p, cudaStream_t s) {
  const unsigned most = std::max<unsigned>(p.nb, 4 * num_sms());
  for (uint32_t part = 0; part < p.slices; part++)
    launch_behind(k_hits, std::min<unsigned>(num_sms() * p.hits_bps, most), 256, 0, s, p, part, p.slices);
}

}  // namespace stc
