// Shared device-side definitions of the GB300 co-occurrence pipeline.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "stc.h"
#include "stc_refmath.h"

#define STC_CLAIM_BIT (1ULL << 63)
#define STC_INIT_LO 100000.0f
#define STC_INIT_HI -100000.0f
#define STC_NONE 0xFFFFFFFFu
#define STC_MAX_LEAF_CAP (1u << 16)    // leaf list capacity bound (tile counts fit in 32 bits)
#define STC_MAX_DEPTH 96            // descent / lookup depth bound
#define STC_PROBE_LIMIT (1ULL << 16)  // longest probe walk before the table counts as full

enum { NODE_INVALID = 0, NODE_BRANCH = 1, NODE_LEAF = 2 };  // index/QTree.h:43-47

// Device error codes (stored in DevState::error, first one wins).
enum {
  ERR_NONE = 0,
  ERR_DESCENT = 1,     // descent reached an invalid node or ran too deep
  ERR_UNITS = 2,       // border checking units exceed refine_size * N
  ERR_PROBE = 3,       // meeting table probe walk exceeded its bound (table full)
  ERR_CAND = 4,        // candidate set / list full
  ERR_DA = 5,          // ordered insertion exceeded its bound
  ERR_EMIT = 6,        // emit buffer full
  ERR_SCHEMA = 7,      // schema or grid stack exhausted
  ERR_LOOKUP = 8,      // border lookup stack overflow
  ERR_BUILD = 9,       // initial quadtree build exceeded capacity
  ERR_MEMTABLE = 10,   // memtable full
  ERR_COMPACT = 11,    // a key to compact lies outside its CTF or names an unknown object
};

// One meeting-table slot (32 B; the reference's meeting_unit of
// tracing/workbench.h:62-83 with the f_box of cuda/geometry.cu).
// While an ordered insertion runs, an empty slot's (start, end) word holds
// the priority of the key claiming it and the key carries STC_CLAIM_BIT.
struct __align__(32) Slot {
  unsigned long long key;
  uint32_t start, end;
  float lo_x, lo_y, hi_x, hi_y;
};

// Distinct keys of one step that were not found by a plain probe.
struct __align__(32) Cand {
  unsigned long long key;
  unsigned long long order;   // first occurrence in the reference's processing order
  float lo_x, lo_y, hi_x, hi_y;
};

// Quadtree node geometry (index/QTree.h:49-62 QTSchema, split in two arrays).
struct __align__(64) Node {
  double mid_x, mid_y, lo_x, lo_y, hi_x, hi_y;
  uint32_t child[4];
};

struct NodeMeta {
  int16_t type, level, overflow, underflow;
  uint32_t grid_id;
  uint32_t parent;
};

// One pair within reach found by the refinement, waiting to be applied to
// the meeting table: the pair (a < b; a = STC_NONE marks an unused place of a
// step that leaves its hits in sequence),
// its priority and its MBR contribution, the box of the two objects' float
// positions of the step (lo = fminf(a's, b's), hi = fmaxf(a's, b's)).
// The key cantor(a, b) is rebuilt when applied. Carrying the box saves the
// table update two dependent random reads of positions per extended meeting.
struct __align__(32) HitRec {
  uint32_t a, b;
  unsigned long long order;  // bit 63: the pair may occur twice this step
  float lo_x, lo_y, hi_x, hi_y;
};

struct __align__(16) U128 {
  unsigned long long lo, hi;
};

// Where a tile of the meeting table keeps its meetings: each in its slot, or
// packed in slot order at the front or the back of the tile, the slots being
// the marks of PipeDev::occ (stc_table.cu).
enum TableLayout : uint32_t { TABLE_SLOTS = 0, TABLE_FRONT = 1, TABLE_BACK = 2 };
constexpr unsigned long long HALO_TOLD = ~0ull;  // the step was told to take the general path
constexpr uint32_t TOLD_STALE = 1u << 31;  // tile_live and occ are not the table's: the step before did not count

// Small device-resident control block.
struct DevState {
  uint32_t schema_stack_index, grids_stack_index;
  uint32_t error, error_info;
  unsigned long long border_units;
  unsigned long long jobs_total;
  unsigned long long tile_load;       // most (occupied slots + hits) of a table tile this step
  unsigned long long cand_count;
  unsigned long long emit_count;      // records in the emit buffer (pending drain)
  unsigned long long tests, exact_tests, hits, ambiguous;
  unsigned long long taken;
  unsigned long long step_emitted;
  unsigned long long halo;            // halo tiles of the step's tiled table update; 0: general path; HALO_TOLD
  uint32_t splits, merges;
  uint32_t told;                      // steps told to be general in a row (PathChoice); TOLD_STALE
  uint32_t overflow_objects;
  uint32_t build_nodes, build_leaves, build_active, build_level;
  uint32_t work_next;                 // generic persistent-kernel work counter
  uint32_t step_t;                    // time of the step in flight (set at its start)
  uint32_t packed;                    // layout of the meeting table's tiles (TableLayout)
  uint32_t redo;                      // a bin overflowed while the tiles were packed (stc_refine.cu, bin_hit)
  unsigned long long hit_count;       // places taken in the hit buffer by a step told to be general
  unsigned long long fast_claims;     // new meetings started this step (claims finalised by the sweep)
  unsigned long long hit_max;         // most hits of a table tile this step
  uint32_t schema_path;               // 1 parallel replay; by one thread: 2 (a cascade, or many events), 0 (asked to)
  uint32_t same_t;                    // the step's time is the last step's
  // memtable (stc_lsm.cu)
  unsigned long long kv_count;        // directed keys in the memtable
  unsigned long long lsm_over_keys;   // keys partitioned to the oversize buffer (flush)
  uint32_t lsm_sid_count;             // objects with at least one key
  uint32_t lsm_over_count;            // the reference's oversize_oid_count
  uint32_t lsm_max_dur, lsm_max_end;  // largest duration / end offset (flush sort widths)
  uint32_t lsm_os_min, lsm_os_max;    // oversize buffer start times (flush)
};

__device__ __forceinline__ void stc_set_error(DevState *st, uint32_t code, uint32_t info) {
  if (atomicCAS(&st->error, 0u, code) == 0u) st->error_info = info;
}

// Float min/max on the IEEE bit pattern (valid for any mix of signs, no NaN).
__device__ __forceinline__ void atomic_min_f(float *a, float v) {
  if (v >= 0.0f) atomicMin((int *)a, __float_as_int(v));
  else atomicMax((unsigned int *)a, __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_f(float *a, float v) {
  if (v >= 0.0f) atomicMax((int *)a, __float_as_int(v));
  else atomicMin((unsigned int *)a, __float_as_uint(v));
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// x % d for a fixed divisor with m = ceil(2^64 / d) (computed on the host):
// the multiply-high quotient is exact or one too large; 64-bit division
// would run through the FP64 pipe.
__device__ __forceinline__ unsigned long long fast_mod(unsigned long long x, unsigned long long d,
                                                       unsigned long long m) {
  unsigned long long q = __umul64hi(x, m);
  unsigned long long r = x - q * d;
  return (long long)r < 0 ? r + d : r;
}

__device__ __forceinline__ bool stc_failed(const DevState *st) {
  return *(volatile const uint32_t *)&st->error != 0u;
}

// Warp-aggregated fetch-add of 1 on a global counter by the lanes that reach
// this call together.
__device__ __forceinline__ unsigned long long agg_inc(unsigned long long *ctr) {
  unsigned m = __activemask();
  unsigned lane = threadIdx.x & 31u;
  int leader = __ffs(m) - 1;
  unsigned long long base = 0;
  if ((int)lane == leader) base = atomicAdd(ctr, (unsigned long long)__popc(m));
  base = __shfl_sync(m, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z ^= z >> 33;
  z *= 0xff51afd7ed558ccdULL;
  z ^= z >> 33;
  z *= 0xc4ceb9fe1a85ec53ULL;
  z ^= z >> 33;
  return z;
}

// Exact integer inverse of the Cantor pairing (util/util.h:72-78 uses a
// double sqrt, which is exact only while 8z+1 < 2^53). 64-bit integer <->
// float conversions run on the FP64 pipe, so the first guess comes from the
// top 32 bits in fp32 (relative error ~2^-22, i.e. a few units for
// v < 2^62); exact integer steps correct it.
__device__ __forceinline__ void cantor_decode(unsigned long long z, uint32_t *a, uint32_t *b) {
  unsigned long long v = 8ULL * z + 1ULL;
  int sh = 64 - __clzll(v);
  sh = sh > 32 ? ((sh - 32 + 1) & ~1) : 0;  // even shift keeps sqrt(v >> sh) * 2^(sh/2)
  float fv = __uint2float_rn((uint32_t)(v >> sh));
  // scale in fp32 before rounding to an integer (r < 2^30 for v < 2^60)
  float rf = sqrtf(fv) * __int_as_float((127 + sh / 2) << 23);
  unsigned long long r = __float2uint_rn(rf);
  while (r * r > v) r--;
  while ((r + 1) * (r + 1) <= v) r++;
  unsigned long long w = (r - 1) / 2;
  unsigned long long t = (w * w + w) / 2;
  *b = (uint32_t)(z - t);
  *a = (uint32_t)(w - (z - t));
}

// metres per degree of longitude at float latitude y (1/dpml), single
// precision; used only by the conservative pre-filter, never for a decision
// by itself.
__device__ __forceinline__ float metres_per_deg_lon_f(float y) {
  float arg = (90.0f - fabsf(y)) * (3.14159265f / 180.0f);
  return sinf(arg) * 111322.2222222f;
}

// An object's float position (the MBR's coordinates).
__device__ __forceinline__ float2 float_pos(double2 q) {
  return make_float2(__double2float_rn(q.x), __double2float_rn(q.y));
}

#define STC_SLAT_F 111322.2222222f   // metres per degree of latitude (1/dpm_lat)
#define STC_SMAX_F 111322.2222222f   // upper bound of metres per degree of longitude

// ---------------------------------------------------------------------------
namespace stc {

// Kernel launches issued by this thread (counted per step in stc_stats).
extern thread_local unsigned long long tl_launches;

// Streaming multiprocessors of the current device
// (cudaDevAttrMultiProcessorCount, looked up once per device): grid-stride
// launches are sized in multiples of it.
int num_sms();

}  // namespace stc

// Prefix for every kernel launch statement: `STC_KL k<<<g, b, 0, s>>>(...);`
#define STC_KL ::stc::tl_launches++,

// Launches a kernel behind the one before it in the stream, without the gap
// between them: its blocks are set up as that one's last blocks end, and wait
// for all of it in after_previous(), which every kernel launched this way
// calls first. A step of 20k objects is 21 short launches: 0.204 -> 0.186 ms;
// 100k 0.142 -> 0.122, 700k 0.291 -> 0.279. (Letting the next kernel's blocks in
// from this one's start holds up its side streams: 700k 0.293, 10M 6.3 -> 6.6.)
template <typename... K, typename... A>
inline void launch_behind(void (*kernel)(K...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 1;
  ::stc::tl_launches++;
  cudaLaunchKernelEx(&c, kernel, K(args)...);
}
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Primitives implemented in stc_sort.cu.
#define STC_SCAN_TILE 2048  // items per scan block
#define STC_RS_TILE 4096    // items per radix-sort block
namespace stc {

// Exclusive scan of n uint32 values (in place allowed). total (device ptr,
// optional) receives the sum as uint64. tmp must hold scan_tmp_words(n) words.
size_t scan_tmp_words(size_t n);
void exclusive_scan_u32(const uint32_t *in, uint32_t *out, size_t n, unsigned long long *total, uint32_t *tmp,
                        cudaStream_t s);

// In-place exclusive scan of nb block sums by one block; total as above.
void scan_sums_u32(uint32_t *sums, size_t nb, unsigned long long *total, cudaStream_t s);

// Stable LSD radix sort of (key, value) uint32 pairs on the low `bits` key
// bits. n_dev (device) holds the item count, n_max bounds it. Result lands
// in (k_out, v_out); k_tmp/v_tmp are scratch of n_max words. hist must hold
// radix_hist_words(n_max) words.
size_t radix_hist_words(size_t n_max);
void radix_sort_u32(const uint32_t *k_in, const uint32_t *v_in, uint32_t *k_out, uint32_t *v_out,
                    uint32_t *k_tmp, uint32_t *v_tmp, const unsigned long long *n_dev, size_t n_max, int bits,
                    uint32_t *hist, uint32_t *scan_tmp, cudaStream_t s);

void iota_u32(uint32_t *out, size_t n, cudaStream_t s);

// Device memory (stc_util.cu). pool_alloc takes it from a pool of the current
// device, in stream order: cudaMalloc and cudaFree of a call's scratch cost
// 0.3 ms each for 300 MB, and stop the device. The pool keeps at most
// POOL_KEEP_BYTES of freed memory and gives it back when an allocation of the
// library fails, when a context of the device is destroyed and in
// stc_release_scratch (pool_release); with the last context the pool goes too.
// dev_malloc is cudaMalloc with a second attempt once the pool is empty. What
// the pool would not keep is taken plainly: a pool maps new gigabytes at a
// quarter of cudaMalloc's rate (8 GB of compaction scratch: 7.3 against 1.1 ms).
constexpr unsigned long long POOL_KEEP_BYTES = 512ull << 20;
constexpr size_t POOL_LARGEST_KEPT = 64u << 20;  // largest single array of a block that is kept for queries
cudaError_t pool_alloc(void **p, size_t bytes, cudaStream_t s);
void pool_free(void *p, cudaStream_t s);
void pool_trim();
void pool_release();
void pool_context(bool begins);  // a context of the current device begins or ends
cudaError_t dev_malloc(void **p, size_t bytes);

// Device scratch of one call on stream s, `total` bytes in all, freed when it
// ends.
class CallScratch {
 public:
  CallScratch(cudaStream_t s, unsigned long long total) : s_(s), pooled_(total <= POOL_KEEP_BYTES) {}
  CallScratch(const CallScratch &) = delete;
  CallScratch &operator=(const CallScratch &) = delete;
  ~CallScratch() {
    for (int i = 0; i < n_; i++) {
      if (pooled_) pool_free(ptr_[i], s_);
      else cudaFree(ptr_[i]);
    }
  }
  template <typename T>
  T *get(size_t count) {
    void *p = nullptr;
    const size_t bytes = (count ? count : 1) * sizeof(T);
    if (error_ == cudaSuccess && n_ == MOST) error_ = cudaErrorMemoryAllocation;
    if (error_ == cudaSuccess) error_ = pooled_ ? pool_alloc(&p, bytes, s_) : dev_malloc(&p, bytes);
    if (error_ != cudaSuccess) return nullptr;
    ptr_[n_++] = p;
    return (T *)p;
  }
  cudaError_t error() const { return error_; }

 private:
  static constexpr int MOST = 40;
  cudaStream_t s_;
  bool pooled_;
  int n_ = 0;
  void *ptr_[MOST];
  cudaError_t error_ = cudaSuccess;
};

// An array of a block kept for queries: cudaFree frees it.
template <typename T>
inline cudaError_t block_alloc(T **p, size_t bytes, cudaStream_t s) {
  return bytes <= POOL_LARGEST_KEPT ? pool_alloc((void **)p, bytes, s) : dev_malloc((void **)p, bytes);
}

}  // namespace stc
