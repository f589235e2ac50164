// Step kernels (a): quadtree partitioning of one step's positions.
//
//   k_descend      phased descent of every point to its leaf, tracking the
//                  deepest ancestor whose box keeps the point away from its
//                  top and right border (tracing/filter.cpp:228-243); leaf
//                  histogram, whose counter also numbers the leaf's members
//   k_leaf_alloc   a range of the member list for every leaf (any order)
//   k_leaf_scatter the leaves' member lists (any order within a leaf)
//   k_leaf_small/big  each leaf's kept members (the first leaf_cap in pid
//                  order, tracing/filter.cpp:95-111) in strip order, their
//                  candidate ranges and the leaf's own refinement jobs
//   k_border_*     depth-first lookup of the top/right leaves within reach of
//                  a border point (tracing/filter.cpp:130-152), counted then
//                  filled in the reference's unit order (pid, then DFS order),
//                  grouped by leaf, and the border units' refinement jobs
//
// Only sets and priorities of the lists matter downstream (a pair's priority
// is its unit's rank and the member's pid, which orders a leaf's members as
// their place in the pid-ordered list does), so leaves get their ranges and
// members their places by atomic counters. Radix sorts of all objects and of
// the border units by leaf, with their scans, took 40 launches a step. One
// GB300, the partition of a step before and now: 20k objects in hotspots 0.24
// and 0.09 ms, 100k uniform objects 0.21 and 0.065, 10M 2.95 and 1.36.
#include <algorithm>

#include "stc_pipeline.cuh"

namespace stc {

static inline unsigned nblk(size_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ double dpml_fast_d(double lat) {
  double absla = fabs(lat);
  if (absla == 90) absla = 89;
  double arg = RN_DIV(RN_MUL(RN_SUB(90.0, absla), STC_REF_PI), 180.0);
  return RN_DIV(360.0, RN_MUL(RN_MUL(sin(arg), 40076.0), 1000.0));
}

// One 32-byte load.
struct __align__(32) Words8 {
  uint32_t v[8];
};
__device__ __forceinline__ Words8 load32(const void *p) {
  Words8 r;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
                 "=r"(r.v[7])
               : "l"(p));
  return r;
}
__device__ __forceinline__ long long word_pair(uint32_t lo, uint32_t hi) {
  return (long long)((unsigned long long)hi << 32 | lo);
}

// One thread per point: from the start of its cell, one 32-byte load a level
// down to the leaf. The deepest ancestor whose box keeps the point away from
// its top and right border (tracing/filter.cpp:228-243) is looked for
// afterwards: the deepest one that does, so a point clear of its leaf's border
// (four of five) is done, the others walk up until they are clear; boxes are
// compared in float offsets from the map's corner, in double within their
// rounding. 10M objects: from the root with every level's node, type and box
// in double 0.77 ms; one load a level 0.60, from the cell's start in double
// 0.71 (both bound by FP64, some 20 operations a point); this form 0.31.
__global__ void __launch_bounds__(256) k_descend(PipeDev p) {
  after_previous();
  uint32_t pid = blockIdx.x * blockDim.x + threadIdx.x;
  if (pid >= p.N) return;
  double2 q;
  if (p.xy_in) {
    q = p.xy_in[pid];
    const_cast<double2 *>(p.xy)[pid] = q;
  } else {
    q = p.xy[pid];
  }
  const uint32_t E = p.sd.start_edge;
  const float rx = __double2float_rn(RN_SUB(q.x, p.sd.ox)), ry = __double2float_rn(RN_SUB(q.y, p.sd.oy));
  const float cx = rx * p.sd.start_sx, cy = ry * p.sd.start_sy;
  const bool inside = cx >= 0.0f && cy >= 0.0f && cx < (float)E && cy < (float)E;
  uint32_t cur = __ldg(&p.sd.start[inside ? (uint32_t)cy * E + (uint32_t)cx : E * E]);
  const long long kx = order_key(__double_as_longlong(q.x)), ky = order_key(__double_as_longlong(q.y));
  for (int d = 0; !(cur & WALK_LEAF) && d < STC_MAX_DEPTH; d++) {
    const Words8 w = load32(&p.sd.walk[cur]);
    const bool right = kx > word_pair(w.v[0], w.v[1]), up = ky > word_pair(w.v[2], w.v[3]);
    cur = up ? (right ? w.v[7] : w.v[6]) : (right ? w.v[5] : w.v[4]);
  }
  const uint32_t gid = cur & ~WALK_LEAF;
  if (!(cur & WALK_LEAF) || gid >= p.G) {
    stc_set_error(p.st, ERR_DESCENT, pid);
    p.leaf_gid[pid] = STC_NONE;
    p.lastvalid[pid] = STC_NONE;
    return;
  }
  p.leaf_gid[pid] = gid;
  p.rank[pid] = atomicAdd(&p.grid_count[gid], 1u);
  uint32_t lv = p.sd.gid_node[gid];
  const uint32_t leaf = lv;
  // (the root is the last resort whether the point is clear of it or not)
  while (lv != 0) {
    const float4 b = p.sd.fbox[lv];
    const float mx = b.z - (rx + p.x_buffer_f), my = b.w - (ry + p.y_buffer_f);
    bool clear;
    if (inside && fminf(fabsf(mx), fabsf(my)) > p.border_eps) {
      clear = mx > 0.0f && my > 0.0f;
    } else {
      const double2 hi = *(const double2 *)&p.sd.nodes[lv].hi_x;
      clear = RN_ADD(q.x, p.x_buffer) < hi.x && RN_ADD(q.y, p.y_buffer) < hi.y;
    }
    if (clear) break;
    lv = p.sd.meta[lv].parent;
  }
  p.lastvalid[pid] = lv != leaf ? lv : STC_NONE;
}

// Per block of 256: each thread's offsets among the block's v[0..K), from
// global counters that move on by the block's totals. Every thread calls it.
// use(sums) runs on thread 0 with the block's totals and puts the counters'
// former values into base.
struct BlockTake {
  uint32_t warp_sum[3][8];
  unsigned long long base[3];
};
template <int K, typename Use>
__device__ __forceinline__ void block_take(const uint32_t (&v)[K], unsigned long long (&at)[K], BlockTake &s, Use use) {
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  uint32_t incl[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    incl[k] = v[k];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl[k], d);
      if ((int)lane >= d) incl[k] += up;
    }
  }
  __syncthreads();  // the last use of s is over
  if (lane == 31)
    for (int k = 0; k < K; k++) s.warp_sum[k][wid] = incl[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t sum[K];
    for (int k = 0; k < K; k++) {
      sum[k] = 0;
      for (int w = 0; w < 8; w++) sum[k] += s.warp_sum[k][w];
    }
    use(sum);
  }
  __syncthreads();
  for (int k = 0; k < K; k++) {
    at[k] = s.base[k] + (incl[k] - v[k]);
    for (uint32_t w = 0; w < wid; w++) at[k] += s.warp_sum[k][w];
  }
}

// Strip order of each leaf's kept members, for the refinement's candidate
// ranges. The leaf is cut into H horizontal strips (H <= STRIPS_MAX) at
// least s_min metres tall, s_min a little above reach. The reference's
// distance takes dy / dpm_lat, a constant scale, so two members within reach
// lie at most one strip apart. Within a strip of at most XSORT_MAX members
// the members are ordered by longitude offset; |dx| * (metres per degree at
// the first point's latitude) <= reach bounds |dx| by wx degrees, wx taken at
// the leaf's smallest scale, so the partners of a member in an ordered strip
// form one window of it, found by binary search. A larger strip (dense
// hotspot leaves at the minimum width, where most pairs are within reach
// anyway) keeps its members unordered and is taken whole.
// Candidates of member i (own rows): the members after it in its strip up
// to its window's end, and its window in the next strip; every pair at most
// a strip apart and within wx is thereby tested once, by its member earlier
// in (strip, longitude) order. Strip and window bounds are computed in fp32
// from the members' leaf offsets; s_min and wx cover their rounding (u times
// the leaf extent) and the scale's with wide margins (2e-4 relative plus 1e-6
// of the leaf extent plus 1-2 mm). The order within a strip only decides
// which member of a pair tests it; each hit's priority comes from the pids.

// Geometry of leaf g with n kept members from `base` on (one thread a leaf: it
// is double arithmetic).
__device__ __forceinline__ LeafGeo leaf_geo(const PipeDev &p, uint32_t g, uint32_t base, uint32_t n) {
  const Node *o = &p.sd.nodes[p.sd.gid_node[g]];
  LeafGeo q;
  q.lo_x = o->lo_x;
  q.lo_y = o->lo_y;
  const double hi_x = o->hi_x, hi_y = o->hi_y;
  const double h_deg = RN_SUB(hi_y, q.lo_y), w_deg = RN_SUB(hi_x, q.lo_x);
  const float h_m = (float)h_deg * STC_SLAT_F, w_m = (float)w_deg * STC_SMAX_F;
  const float s_min = p.reach_f * 1.0001f + 1e-6f * h_m + 1e-3f;
  float hf = floorf(h_m / s_min);
  q.strips = hf < 1.0f ? 1u : (hf > (float)STRIPS_MAX ? STRIPS_MAX : (uint32_t)hf);
  q.inv = q.strips > 1 ? (float)q.strips / (float)h_deg : 0.0f;  // strips per degree from the low edge
  // smallest metres per degree of longitude of any first point of a pair
  // (the leaf's latitudes, widened by 1e-3 degrees for border points)
  const double lat = fmax(fabs(q.lo_y), fabs(hi_y)) + 1e-3;
  const float s_lon = metres_per_deg_lon_f(__double2float_rn(lat < 89.0 ? lat : 89.0)) * (1.0f - 1e-5f);
  q.wx = (p.reach_f * 1.0002f + 1e-6f * (w_m + h_m) + 2e-3f) / s_lon;
  q.ext_x = (float)w_deg;
  q.ext_y = (float)h_deg;
  q.base = base;
  q.n = n;
  return q;
}

// A range of the member list for each leaf, and its geometry.
__global__ void __launch_bounds__(256) k_leaf_alloc(PipeDev p) {
  after_previous();
  __shared__ BlockTake s;
  const uint32_t ids = p.sd.high[1];
  for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < ids; g0 += gridDim.x * blockDim.x) {
    const uint32_t g = g0 + threadIdx.x;
    const uint32_t cnt = g < ids ? p.grid_count[g] : 0u;
    const uint32_t n = cnt < p.leaf_cap ? cnt : p.leaf_cap;
    const uint32_t v[3] = {cnt, n && n <= LEAF_SMALL ? 1u : 0u, n > LEAF_SMALL ? 1u : 0u};
    unsigned long long at[3];
    block_take(v, at, s, [&](const uint32_t (&sum)[3]) {
      for (int k = 0; k < 3; k++)
        s.base[k] = sum[k] ? atomicAdd(&p.ctr[k == 0 ? CTR_MEMBERS : k == 1 ? CTR_SMALL : CTR_BIG],
                                       (unsigned long long)sum[k]) : 0ull;
    });
    if (!cnt) continue;
    p.grid_start[g] = (uint32_t)at[0];
    p.lgeo[g] = leaf_geo(p, g, (uint32_t)at[0], n);
    if (n <= LEAF_SMALL) p.leaf_list[at[1]] = g;
    else p.leaf_list[p.leaves_max - 1 - at[2]] = g;  // big leaves from the list's end
    if (cnt > n) atomicAdd(&p.st->overflow_objects, cnt - n);
  }
}

__global__ void __launch_bounds__(256) k_leaf_scatter(PipeDev p) {
  after_previous();
  const uint32_t pid = blockIdx.x * blockDim.x + threadIdx.x;
  if (pid >= p.N) return;
  const uint32_t g = p.leaf_gid[pid];
  if (g != STC_NONE) p.lpid[p.grid_start[g] + p.rank[pid]] = pid;
}

__device__ __forceinline__ uint32_t member_strip(float ly, float inv, uint32_t H) {
  float c = floorf(ly * inv);
  c = fminf(fmaxf(c, 0.0f), (float)(H - 1));
  return (uint32_t)c;
}

// First index in [lo, hi) of a longitude-ordered strip whose offset is
// greater than x (upper = true) or not below x (upper = false). at(i): the
// offset of member i.
template <typename At>
__device__ __forceinline__ uint32_t x_bound(At at, uint32_t lo, uint32_t hi, float x, bool upper) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    const float v = at(mid);
    if (upper ? v <= x : v < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Candidate ranges of member i in strip sidx (start[s]: first member of strip
// s, start[H] = n); returns how many candidates they hold.
template <typename At>
__device__ __forceinline__ uint32_t member_window(At at, const uint32_t *start, uint32_t H, uint32_t sidx, uint32_t i,
                                                  float wx, uint2 &cand) {
  const float xi = at(i);
  const uint32_t en = start[sidx + 1];
  const uint32_t e1 = en - start[sidx] <= XSORT_MAX ? x_bound(at, i + 1, en, xi + wx, true) : en;
  uint32_t a2 = 0, b2 = 0;
  if (sidx + 1 < H) {
    const uint32_t en2 = start[sidx + 2];
    a2 = en;
    b2 = en2;
    if (en2 - en <= XSORT_MAX) {
      a2 = x_bound(at, en, en2, xi - wx, false);
      b2 = x_bound(at, a2, en2, xi + wx, true);
    }
  }
  cand = make_uint2(e1 | a2 << 16, b2);
  return (e1 - (i + 1)) + (b2 - a2);
}

// Refinement jobs of one leaf, written by `threads` threads (thread `me`):
// rows row blocks with `chunks` candidate chunks each, one job per chunk while
// the list has room to spare (p.jobs_extra), else one per row block. head: a
// broadcast slot in shared memory.
struct JobHead {
  unsigned long long at;
  uint32_t split;
};
__device__ __forceinline__ JobHead take_jobs(const PipeDev &p, uint32_t rows, uint32_t chunks) {
  const unsigned long long extra = (unsigned long long)rows * (chunks - 1);
  JobHead h;
  h.split = !extra || atomicAdd(&p.ctr[CTR_EXTRA], extra) + extra <= p.jobs_extra;
  h.at = atomicAdd(&p.st->jobs_total, h.split ? rows + extra : (unsigned long long)rows);
  return h;
}
__device__ __forceinline__ void write_jobs(const PipeDev &p, const JobHead &h, uint32_t g, uint32_t own, uint32_t rows,
                                           uint32_t chunks, uint32_t me, uint32_t threads) {
  const uint32_t total = h.split ? rows * chunks : rows;
  for (uint32_t e = me; e < total; e += threads)
    p.jobs[h.at + e] = h.split ? make_uint4(g, e / chunks | own, e % chunks, 1u) : make_uint4(g, e | own, 0u, chunks);
}

// The leaf's members: its list, or, of a leaf with more than leaf_cap, the
// leaf_cap lowest pids (tracing/filter.cpp:100-104), found by a radix select
// of the block and copied aside. hist: 256 words, var: 3 words.
__device__ const uint32_t *kept_members(const PipeDev &p, uint32_t base, uint32_t cnt, uint32_t *hist, uint32_t *var) {
  const uint32_t *list = p.lpid + base;
  if (cnt <= p.leaf_cap) return list;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    var[0] = 0;           // the bits known of the last pid kept
    var[1] = p.leaf_cap;  // its place among those sharing them
    var[2] = 0;
  }
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (uint32_t k = tid; k < 256; k += blockDim.x) hist[k] = 0;
    __syncthreads();
    const uint32_t mask = shift == 24 ? 0u : 0xFFFFFFFFu << (shift + 8), known = var[0];
    for (uint32_t i = tid; i < cnt; i += blockDim.x)
      if ((list[i] & mask) == known) atomicAdd(&hist[(list[i] >> shift) & 255u], 1u);
    __syncthreads();
    if (tid == 0) {
      uint32_t need = var[1], b = 0;
      while (b < 255u && hist[b] < need) need -= hist[b++];
      var[0] = known | b << shift;
      var[1] = need;
    }
    __syncthreads();
  }
  const uint32_t lastp = var[0];
  for (uint32_t i = tid; i < cnt; i += blockDim.x)
    if (list[i] <= lastp) p.lpid2[base + atomicAdd(&var[2], 1u)] = list[i];
  __syncthreads();
  return p.lpid2 + base;
}

// Leaves of up to LEAF_SMALL kept members: a block each, two members a
// thread, the strip counting sort, the longitude ranks and the windows in
// shared memory. (A warp a leaf took its strips one after the other: 53 us
// whatever the object count, 0.57 ms at 10M objects and 0.42 for the gather
// before it; this form 8 us and 0.44 for both.)
__global__ void __launch_bounds__(LEAF_SMALL / 2, 12) k_leaf_small(PipeDev p) {
  after_previous();
  constexpr uint32_t T = LEAF_SMALL / 2;
  __shared__ uint32_t start[STRIPS_MAX + 2], hist[256], var[3], longest;
  __shared__ float sx[LEAF_SMALL], fx[LEAF_SMALL];  // offsets in (strip, arrival) and in final order
  __shared__ uint8_t fs[LEAF_SMALL];                // strips in final order
  __shared__ JobHead head;
  const uint32_t tid = threadIdx.x, lane = lane_id();
  const uint32_t leaves = (uint32_t)p.ctr[CTR_SMALL];
  for (uint32_t li = blockIdx.x; li < leaves; li += gridDim.x) {
    const uint32_t g = p.leaf_list[li];
    const LeafGeo q = p.lgeo[g];
    const uint32_t H = q.strips, n = q.n, base = q.base;
    const uint32_t *list = kept_members(p, base, p.grid_count[g], hist, var);
    for (uint32_t k = tid; k < STRIPS_MAX + 2; k += T) start[k] = 0;
    if (tid == 0) longest = 0;
    __syncthreads();
    float4 v[2];
    float2 f[2];
    uint32_t sidx[2], rk[2];
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const uint32_t i = tid + m * T;
      if (i >= n) continue;
      const uint32_t pid = list[i];
      const double2 xy = p.xy[pid];
      f[m] = float_pos(xy);
      v[m] = make_float4(__double2float_rn(RN_SUB(xy.x, q.lo_x)), __double2float_rn(RN_SUB(xy.y, q.lo_y)),
                         metres_per_deg_lon_f(f[m].y), __uint_as_float(pid));
      sidx[m] = member_strip(v[m].y, q.inv, H);
      rk[m] = atomicAdd(&start[sidx[m] + 1], 1u);
    }
    __syncthreads();
    if (tid < 32) {  // start[s] = members before strip s: a scan of the 64 counts, two a lane
      const uint32_t c0 = start[2 * lane + 1], c1 = start[2 * lane + 2];
      uint32_t x = c0 + c1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if ((int)lane >= d) x += y;
      }
      __syncwarp();
      start[2 * lane + 1] = x - c1;
      start[2 * lane + 2] = x;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; m++)
      if (tid + m * T < n) sx[start[sidx[m]] + rk[m]] = v[m].x;
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; m++) {
      if (tid + m * T >= n) continue;
      const uint32_t st = start[sidx[m]], en = start[sidx[m] + 1], at = st + rk[m];
      uint32_t k = at;
      if (en - st <= XSORT_MAX) {  // place by longitude
        k = st;
        for (uint32_t b = st; b < en; b++) k += (sx[b] < v[m].x || (sx[b] == v[m].x && b < at)) ? 1u : 0u;
      }
      fx[k] = v[m].x;
      fs[k] = (uint8_t)sidx[m];
      p.spts[base + k] = v[m];
      p.sfxy[base + k] = f[m];
    }
    __syncthreads();
    uint32_t most = 0;
    for (uint32_t i = tid; i < n; i += T) {
      uint2 c;
      most = max(most, member_window([&](uint32_t k) { return fx[k]; }, start, H, fs[i], i, q.wx, c));
      p.scand[base + i] = c;
    }
    if (most) atomicMax(&longest, most);
    for (uint32_t k = tid; k <= H; k += T) p.sstart[(size_t)g * STRIP_STRIDE + k] = (uint16_t)start[k];
    __syncthreads();
    const uint32_t chunks = max(1u, (longest + p.refine_chunk - 1) / p.refine_chunk), rows = (n + 31) / 32;
    if (tid == 0) head = take_jobs(p, rows, chunks);
    __syncthreads();
    write_jobs(p, head, g, JOB_OWN, rows, chunks, tid, T);
  }
}

// Larger leaves: a block of 512 each, members in device memory.
__global__ void __launch_bounds__(512) k_leaf_big(PipeDev p) {
  after_previous();
  constexpr uint32_t T = 512;
  __shared__ uint32_t start[STRIPS_MAX + 2], hist[256], var[3], longest;
  __shared__ JobHead head;
  const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const uint32_t leaves = (uint32_t)p.ctr[CTR_BIG];
  for (uint32_t li = blockIdx.x; li < leaves; li += gridDim.x) {
    const uint32_t g = p.leaf_list[p.leaves_max - 1 - li];
    const LeafGeo q = p.lgeo[g];
    const uint32_t H = q.strips, n = q.n, base = q.base;
    const uint32_t *list = kept_members(p, base, p.grid_count[g], hist, var);
    for (uint32_t k = tid; k < STRIPS_MAX + 2; k += T) start[k] = 0;
    if (tid == 0) longest = 0;
    __syncthreads();
    uint32_t *place = p.rank + base;  // (strip << 16 | number within strip); the ranks are no longer needed
    for (uint32_t i = tid; i < n; i += T) {
      const uint32_t pid = list[i];
      const double2 xy = p.xy[pid];
      const float ly = __double2float_rn(RN_SUB(xy.y, q.lo_y));
      p.pts[base + i] = make_float4(__double2float_rn(RN_SUB(xy.x, q.lo_x)), ly,
                                    metres_per_deg_lon_f(__double2float_rn(xy.y)), __uint_as_float(pid));
      const uint32_t sidx = member_strip(ly, q.inv, H);
      place[i] = sidx << 16 | atomicAdd(&start[sidx + 1], 1u);
    }
    __syncthreads();
    if (tid < 32) {
      const uint32_t c0 = start[2 * lane + 1], c1 = start[2 * lane + 2];
      uint32_t x = c0 + c1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if ((int)lane >= d) x += y;
      }
      __syncwarp();
      start[2 * lane + 1] = x - c1;
      start[2 * lane + 2] = x;
    }
    __syncthreads();
    for (uint32_t i = tid; i < n; i += T) {
      const uint32_t u = place[i], k = start[u >> 16] + (u & 0xFFFFu);
      const float4 v = p.pts[base + i];
      p.spts[base + k] = v;
      p.sfxy[base + k] = float_pos(p.xy[__float_as_uint(v.w)]);
    }
    __syncthreads();
    // strips of 2 to XSORT_MAX members in longitude order, a warp a strip:
    // each member's rank among the strip's (offset, position) pairs, its
    // elements in four slots of 32 lanes
    for (uint32_t sidx = warp; sidx < H; sidx += T / 32) {
      const uint32_t st = start[sidx], L = start[sidx + 1] - st;
      if (L > XSORT_MAX || L < 2) continue;
      const uint32_t slots = (L + 31) / 32;
      float4 v[4];
      float2 f[4];
      uint32_t rk[4] = {0, 0, 0, 0};
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const uint32_t e = lane + 32u * m;
        v[m] = e < L ? p.spts[base + st + e] : make_float4(0.f, 0.f, 0.f, 0.f);
        f[m] = e < L ? p.sfxy[base + st + e] : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int m2 = 0; m2 < 4; m2++) {
        if ((uint32_t)m2 >= slots) break;
        for (uint32_t src = 0; src < 32; src++) {
          const float xb = __shfl_sync(0xffffffffu, v[m2].x, src);
          const uint32_t b = src + 32u * m2;
          if (b >= L) break;
#pragma unroll
          for (int m = 0; m < 4; m++) {
            const uint32_t a = lane + 32u * m;
            rk[m] += (xb < v[m].x || (xb == v[m].x && b < a)) ? 1u : 0u;
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const uint32_t e = lane + 32u * m;
        if (e < L) {
          p.spts[base + st + rk[m]] = v[m];
          p.sfxy[base + st + rk[m]] = f[m];
        }
      }
    }
    __syncthreads();
    uint32_t most = 0;
    const float4 *lp = p.spts + base;
    for (uint32_t i = tid; i < n; i += T) {
      uint32_t lo = 0, hi = H;  // the member's strip: start[lo] <= i < start[hi]
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (start[mid] <= i) lo = mid; else hi = mid;
      }
      uint2 c;
      most = max(most, member_window([&](uint32_t k) { return lp[k].x; }, start, H, lo, i, q.wx, c));
      p.scand[base + i] = c;
    }
    if (most) atomicMax(&longest, most);
    for (uint32_t k = tid; k <= H; k += T) p.sstart[(size_t)g * STRIP_STRIDE + k] = (uint16_t)start[k];
    __syncthreads();
    const uint32_t chunks = max(1u, (longest + p.refine_chunk - 1) / p.refine_chunk), rows = (n + 31) / 32;
    if (tid == 0) head = take_jobs(p, rows, chunks);
    __syncthreads();
    write_jobs(p, head, g, JOB_OWN, rows, chunks, tid, T);
  }
}

// box::distance(p, geography=true) <= reach (geometry/geometry.h:174-185),
// decided exactly: fp64 containment and degree offsets as in the reference,
// then the metric step in fp32 with a +-64 u relative band (u = 2^-24), then
// the reference's fp64 division and square root, and within 1e-12 of reach
// the correctly rounded sine.
__device__ bool box_within_exact(const Node &c, double x, double y, double reach, float reach_f, float s_lon,
                                 double &dp_fast) {
  if (x >= c.lo_x && x <= c.hi_x && y >= c.lo_y && y <= c.hi_y) return true;  // distance 0
  double dx = RN_SUB(fabs(RN_SUB(x, RN_MUL(RN_ADD(c.lo_x, c.hi_x), 0.5))), RN_MUL(RN_SUB(c.hi_x, c.lo_x), 0.5));
  double dy = RN_SUB(fabs(RN_SUB(y, RN_MUL(RN_ADD(c.lo_y, c.hi_y), 0.5))), RN_MUL(RN_SUB(c.hi_y, c.lo_y), 0.5));
  if (dx < 0.0) dx = 0.0;
  if (dy < 0.0) dy = 0.0;
  float fx = __double2float_rn(dx) * s_lon, fy = __double2float_rn(dy) * STC_SLAT_F;
  float d2 = fx * fx + fy * fy;
  const float lo = reach_f * (1.0f - 64.0f * 5.9604645e-08f), hi = reach_f * (1.0f + 64.0f * 5.9604645e-08f);
  if (d2 <= lo * lo) return true;
  if (d2 >= hi * hi) return false;
  if (dp_fast == 0.0) dp_fast = dpml_fast_d(y);
  double d = stc_box_distance_ref(c.lo_x, c.lo_y, c.hi_x, c.hi_y, x, y, dp_fast);
  if (fabs(d - reach) > 1e-12 * reach) return d <= reach;
  return stc_box_distance_ref(c.lo_x, c.lo_y, c.hi_x, c.hi_y, x, y, stc_dpml_ref(y)) <= reach;
}

// Lookup of one border point (tracing/filter.cpp:130-152): depth-first from
// last_valid over children 0..3, collecting the leaves within reach that lie
// above the point or to its right. Node distances are first classified in
// fp32 from map-relative float boxes; the band of width border_delta around
// reach (bounding the fp32 rounding of the offsets, see stc_create) goes to
// box_within_exact. Writes the first `keep` leaf ids to out; returns the
// count, or 0xFFFFFFFF on stack overflow.
// A node's four children are classified together, from its own box and split
// point (two loads a node opened), and the ones within reach stacked in
// reverse, so that they come off in depth-first order: a pop is a leaf of the
// result, or a node to open. A child's box is its parent's cut at the split
// point; its stored corners may differ from that by a double's last place,
// which the band covers many times over. (Child after child, each with loads
// of its own and its box in double: 0.67 ms at 10M objects; this form 0.42.)
#define LOOKUP_DEPTH 64                    // levels below the start
#define LOOKUP_STACK (3 * LOOKUP_DEPTH + 8)
// Metres of v outside [lo, hi], squared.
__device__ __forceinline__ float outside2(float v, float lo, float hi, float scale) {
  const float c = (lo + hi) * 0.5f, hw = (hi - lo) * 0.5f;
  const float d = fmaxf(fabsf(v - c) - hw, 0.0f) * scale;
  return d * d;
}

__device__ uint32_t border_lookup(const PipeDev &p, uint32_t pid, uint32_t lv, uint32_t *out, uint32_t keep) {
  double2 q = p.xy[pid];
  float px = __double2float_rn(RN_SUB(q.x, p.sd.ox)), py = __double2float_rn(RN_SUB(q.y, p.sd.oy));
  float s_lon = metres_per_deg_lon_f(__double2float_rn(q.y));
  float reach_f = p.reach_f;
  float rlo = fmaxf(reach_f - p.border_delta, 0.0f), rhi = reach_f + p.border_delta;
  float rlo2 = rlo * rlo, rhi2 = rhi * rhi;
  // the fp32 band only covers points inside the map box (offsets bounded by its extent)
  bool fast_ok = q.x >= p.map_lo_x && q.x <= p.map_hi_x && q.y >= p.map_lo_y && q.y <= p.map_hi_y;
  double dpf = 0.0;
  uint32_t stk[LOOKUP_STACK];
  int sp = 1;
  stk[0] = lv;
  uint32_t cnt = 0;
  while (sp > 0) {
    const uint32_t top = stk[--sp];
    if (top & WALK_LEAF) {
      if (cnt < keep) out[cnt] = top & ~WALK_LEAF;
      cnt++;
      continue;
    }
    if (sp + 4 > LOOKUP_STACK) return 0xFFFFFFFFu;
    const Words8 wb = load32(&p.sd.wbox[top]);
    const uint4 c4 = *(const uint4 *)p.sd.walk[top].child;
    const float4 b = make_float4(__uint_as_float(wb.v[0]), __uint_as_float(wb.v[1]), __uint_as_float(wb.v[2]),
                                 __uint_as_float(wb.v[3]));
    const float mx = __uint_as_float(wb.v[4]), my = __uint_as_float(wb.v[5]);
    const float dx2[2] = {outside2(px, b.x, mx, s_lon), outside2(px, mx, b.z, s_lon)};
    const float dy2[2] = {outside2(py, b.y, my, STC_SLAT_F), outside2(py, my, b.w, STC_SLAT_F)};
#pragma unroll
    for (int i = 3; i >= 0; i--) {
      const float d2 = dx2[i & 1] + dy2[i >> 1];
      int decided = !fast_ok ? 0 : d2 <= rlo2 ? 1 : (d2 >= rhi2 ? -1 : 0);  // 1 within, -1 outside
      if (decided < 0) continue;
      const uint32_t ch = i == 0 ? c4.x : i == 1 ? c4.y : i == 2 ? c4.z : c4.w;
      const bool leaf = (ch & WALK_LEAF) != 0;
      // the leaf lies above, or to the right within the point's row: decided
      // on floats, the exact box fetched only within their rounding
      int wanted = 1;
      if (leaf) {
        const float lx = (i & 1) ? mx : b.x, ly = (i >> 1) ? my : b.y, hy = (i >> 1) ? b.w : my;
        const int above = py < ly - p.border_eps ? 1 : (py > ly + p.border_eps ? -1 : 0);
        const int below_top = py < hy - p.border_eps ? 1 : (py > hy + p.border_eps ? -1 : 0);
        const int right = px < lx - p.border_eps ? 1 : (px > lx + p.border_eps ? -1 : 0);
        const int row = below_top < 0 || right < 0 ? -1 : (below_top > 0 && right > 0 ? 1 : 0);
        wanted = above > 0 || row > 0 ? 1 : (above < 0 && row < 0 ? -1 : 0);
        if (!fast_ok) wanted = 0;
      }
      if (wanted < 0) continue;
      if (decided == 0 || wanted == 0) {
        const Node &c = p.sd.nodes[leaf ? p.sd.gid_node[ch & ~WALK_LEAF] : ch];
        if (decided == 0 && !box_within_exact(c, q.x, q.y, p.reach, reach_f, s_lon, dpf)) continue;
        if (leaf && !(q.y < c.lo_y || (q.y < c.hi_y && q.x < c.lo_x))) continue;
      }
      stk[sp++] = ch;
    }
  }
  return cnt;
}

#define BORDER_KEEP 4

// Border units of the points of a block's TILE pids: their lookups packed
// together, then each point's offset within the block. T threads: a quarter of
// TILE where that fills the GPU, TILE where all points have room for a thread
// of their own at once (a lookup is a chain of dependent loads, and a dense
// crowd's tile has two or three a thread: the wait for the border units of 20k objects in
// hotspots 43 -> 25 us a step, of 60k 41 -> 14).
template <uint32_t TILE, uint32_t T>
__global__ void __launch_bounds__(T, 1024 / T) k_border_count(PipeDev p) {
  __shared__ __align__(16) uint32_t cnts[TILE];
  __shared__ uint16_t list[TILE];
  __shared__ uint32_t nlist, warp_sum[TILE / 128];
  const uint32_t tid = threadIdx.x, lane = lane_id(), first = blockIdx.x * TILE;
  if (tid == 0) nlist = 0;
  __syncthreads();
  for (uint32_t i = tid; i < TILE; i += T) {
    cnts[i] = 0;
    const bool border = first + i < p.N && p.lastvalid[first + i] != STC_NONE;
    const uint32_t ball = __ballot_sync(0xffffffffu, border);
    uint32_t at = 0;
    if (lane == 0 && ball) at = atomicAdd(&nlist, (uint32_t)__popc(ball));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(ball & ((1u << lane) - 1u));
    if (border) list[at] = (uint16_t)i;
  }
  __syncthreads();
  for (uint32_t i = tid; i < nlist; i += T) {
    const uint32_t k = list[i], pid = first + k;
    uint32_t *out = p.bres + (size_t)BORDER_KEEP * pid, keep = BORDER_KEEP, c = 0;
    for (;;) {
      c = border_lookup(p, pid, p.lastvalid[pid], out, keep);
      if (c == 0xFFFFFFFFu) {
        stc_set_error(p.st, ERR_LOOKUP, pid);
        c = 0;
      }
      if (c <= keep) break;
      // rare: more leaves than bres holds for a point go to a pool (more than
      // the pool holds are more units than there may be, which is reported)
      const unsigned long long at = atomicAdd(&p.ctr[CTR_POOL], (unsigned long long)c);
      if (at + c > p.U_cap) {
        p.bres[(size_t)BORDER_KEEP * pid] = STC_NONE;
        break;
      }
      p.bres[(size_t)BORDER_KEEP * pid] = (uint32_t)at;
      out = p.bu_sorted_pos + at;  // free until the units are grouped
      keep = c;
    }
    cnts[k] = c;
  }
  __syncthreads();
  // four consecutive points a thread
  uint4 c = make_uint4(0, 0, 0, 0);
  if (tid < TILE / 4) c = ((const uint4 *)cnts)[tid];
  const uint32_t sum = c.x + c.y + c.z + c.w;
  uint32_t incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
    if ((int)lane >= d) incl += up;
  }
  if (lane == 31 && tid < TILE / 4) warp_sum[tid >> 5] = incl;
  __syncthreads();
  if (tid >= TILE / 4) return;
  uint32_t before = incl - sum;
  for (uint32_t w = 0; w < (tid >> 5); w++) before += warp_sum[w];
  const uint32_t pid = first + 4 * tid;
  const uint32_t cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (pid + k < p.N) {
      p.bcount[pid + k] = cc[k];
      p.boff[pid + k] = before;
    }
    before += cc[k];
  }
  if (tid == TILE / 4 - 1) p.bsum[blockIdx.x] = before;
}

// The units in the reference's order, and each unit's number within its leaf.
__global__ void __launch_bounds__(256) k_border_fill(PipeDev p) {
  after_previous();
  const uint32_t pid = blockIdx.x * blockDim.x + threadIdx.x;
  if (pid == 0 && p.st->border_units >= p.U_cap) stc_set_error(p.st, ERR_UNITS, (uint32_t)p.st->border_units);
  if (pid >= p.N) return;
  const uint32_t c = p.bcount[pid];
  if (!c) return;
  const unsigned long long base = (unsigned long long)p.boff[pid] + p.bsum[pid / p.border_tile];
  p.boff[pid] = (uint32_t)base;
  if (base + c > p.U_cap) return;  // reported above
  const uint32_t *src = p.bres + (size_t)BORDER_KEEP * pid;
  if (c > BORDER_KEEP) {  // in the pool
    if (*src == STC_NONE) return;
    src = p.bu_sorted_pos + *src;
  }
  for (uint32_t k = 0; k < c; k++) {
    const uint32_t gid = src[k];
    p.bu_gid[base + k] = gid;
    p.bu_pid[base + k] = pid;
    p.bu_rank[base + k] = atomicAdd(&p.bu_cnt[gid], 1u);
  }
}

// A range of the grouped units for every leaf that has some, and their jobs:
// 32 units against one chunk of refine_chunk positions of the leaf's members
// (a unit's ranges hold at most all of them).
__global__ void __launch_bounds__(256) k_border_alloc(PipeDev p) {
  after_previous();
  __shared__ BlockTake s;
  __shared__ uint32_t split;
  const uint32_t lane = lane_id(), ids = p.sd.high[1];
  for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < ids; g0 += gridDim.x * blockDim.x) {
    const uint32_t g = g0 + threadIdx.x;
    const uint32_t m = g < ids ? p.bu_cnt[g] : 0u;
    uint32_t rows = 0, chunks = 1;
    if (m) {
      const uint32_t cnt = p.grid_count[g], n = cnt < p.leaf_cap ? cnt : p.leaf_cap;
      if (n) {
        rows = (m + 31) / 32;
        chunks = (n + p.refine_chunk - 1) / p.refine_chunk;
      }
    }
    // units, row blocks, jobs beyond one per row block; the block's leaves are
    // cut into chunks together, or not at all
    const uint32_t v[3] = {m, rows, jobs_beyond(rows, chunks, p.jobs_extra)};
    unsigned long long at[3];
    block_take(v, at, s, [&](const uint32_t (&sum)[3]) {
      s.base[0] = sum[0] ? atomicAdd(&p.ctr[CTR_UNITS], (unsigned long long)sum[0]) : 0ull;
      split = !sum[2] || atomicAdd(&p.ctr[CTR_EXTRA], (unsigned long long)sum[2]) + sum[2] <= p.jobs_extra;
      s.base[1] = sum[1] ? atomicAdd(&p.st->jobs_total, (unsigned long long)sum[1] + (split ? sum[2] : 0u)) : 0ull;
      s.base[2] = 0;
    });
    if (m) p.bu_start[g] = (uint32_t)at[0];
    JobHead h;
    h.split = split;
    h.at = at[1] + (split ? at[2] : 0ull);
    // the warp writes its leaves' jobs together, one leaf after the other
    for (uint32_t todo = __ballot_sync(0xffffffffu, rows != 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      JobHead hh = h;
      hh.at = __shfl_sync(0xffffffffu, h.at, src);
      write_jobs(p, hh, __shfl_sync(0xffffffffu, g, src), 0u, __shfl_sync(0xffffffffu, rows, src),
                 __shfl_sync(0xffffffffu, chunks, src), lane, 32);
    }
  }
}

__global__ void __launch_bounds__(256) k_border_scatter(PipeDev p) {
  after_previous();
  const unsigned long long n = p.st->border_units < p.U_cap ? p.st->border_units : 0ull;
  for (unsigned long long u = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (unsigned long long)gridDim.x * blockDim.x)
    p.bu_sorted_pos[p.bu_start[p.bu_gid[u]] + p.bu_rank[u]] = (uint32_t)u;
}

void step_descend(PipeDev &p, cudaStream_t s) { launch_behind(k_descend, nblk(p.N), 256, 0, s, p); }

void step_leaves(PipeDev &p, cudaStream_t s) {
  launch_behind(k_leaf_alloc, std::min<unsigned>(nblk(p.G), num_sms() * 4), 256, 0, s, p);
  launch_behind(k_leaf_scatter, nblk(p.N), 256, 0, s, p);
  launch_behind(k_leaf_small, num_sms() * 12, LEAF_SMALL / 2, 0, s, p);
  if (p.leaf_cap > LEAF_SMALL) launch_behind(k_leaf_big, num_sms() * 2, 512, 0, s, p);
}

void step_border(PipeDev &p, cudaStream_t s) {
  const unsigned tiles = nblk(p.N, p.border_tile);
  if (p.border_tile == 1024) STC_KL k_border_count<1024, 256><<<tiles, 256, 0, s>>>(p);
  else if (p.N > num_sms() * 1024u) STC_KL k_border_count<256, 64><<<tiles, 64, 0, s>>>(p);
  else STC_KL k_border_count<256, 256><<<tiles, 256, 0, s>>>(p);
  scan_sums_u32(p.bsum, tiles, &p.st->border_units, s);
  launch_behind(k_border_fill, nblk(p.N), 256, 0, s, p);
  launch_behind(k_border_alloc, std::min<unsigned>(nblk(p.G), num_sms() * 4), 256, 0, s, p);
  launch_behind(k_border_scatter, std::min<unsigned>(nblk(p.N), num_sms() * 16), 256, 0, s, p);
}

}  // namespace stc
