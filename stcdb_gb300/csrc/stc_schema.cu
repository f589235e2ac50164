// Quadtree schema: GPU build and per-step dynamic update.
//
// Build (index/QTree.h:157-311, tracing/filter.cpp:27-93): the reference
// inserts points one by one and splits a leaf as soon as it holds
// grid_capacity objects and width(true)/2 > reach. Objects only ever get
// added, so the final tree does not depend on insertion order: a node is
// split iff the number of step-0 points that descend into it is at least
// grid_capacity and the width condition holds. The build therefore runs level
// by level (count points per node of the level, decide splits, move points
// to children), then numbers nodes in preorder with children 0..3
// (QTNode::create_schema) and leaves in depth-first order (QTNode::set_id).
//
// Update (tracing/filter.cpp:316-449): the reference visits nodes 0..S-1 in
// order. Phase 1 evaluates every node in parallel against the pre-sweep
// state; the only way an earlier visit changes a later decision is a merge
// that turns a branch into a leaf before its parent (higher index) is
// visited, so phase 2 replays the flagged events in index order on one
// thread, with those parents queued for re-evaluation at their own index.
// Stack pops and pushes happen in exactly the reference's order.
#include <algorithm>
#include <vector>

#include "stc_schema.cuh"

namespace stc {

__device__ __forceinline__ double dpml_fast(double lat) {
  double absla = fabs(lat);
  if (absla == 90) absla = 89;
  double arg = RN_DIV(RN_MUL(RN_SUB(90.0, absla), STC_REF_PI), 180.0);
  return RN_DIV(360.0, RN_MUL(RN_MUL(sin(arg), 40076.0), 1000.0));
}

// Geographic width of a box (geometry/geometry.h:166-172), returning the
// value computed with the correctly rounded sine whenever the comparison
// against thr could depend on the last bits of the fast one.
__device__ double width_geo(double lx, double ly, double hx, double thr) {
  double w = RN_DIV(RN_SUB(hx, lx), dpml_fast(ly));
  if (fabs(w - thr) > 1e-12 * fabs(thr)) return w;
  return RN_DIV(RN_SUB(hx, lx), stc_dpml_ref(ly));
}

__device__ __forceinline__ void set_child_box(Node &c, const Node &p, int i) {
  // QTNode::split children (index/QTree.h:163-166)
  double lx = (i & 1) ? p.mid_x : p.lo_x;
  double hx = (i & 1) ? p.hi_x : p.mid_x;
  double ly = (i & 2) ? p.mid_y : p.lo_y;
  double hy = (i & 2) ? p.hi_y : p.mid_y;
  c.lo_x = lx; c.lo_y = ly; c.hi_x = hx; c.hi_y = hy;
  c.mid_x = RN_DIV(RN_ADD(hx, lx), 2.0);
  c.mid_y = RN_DIV(RN_ADD(hy, ly), 2.0);
  c.child[0] = c.child[1] = c.child[2] = c.child[3] = STC_NONE;
}

__global__ void k_build_root(Node *bn, NodeMeta *bm, double lx, double ly, double hx, double hy, uint32_t *node_of,
                             uint32_t n, DevState *st) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    Node r;
    r.lo_x = lx; r.lo_y = ly; r.hi_x = hx; r.hi_y = hy;
    r.mid_x = RN_DIV(RN_ADD(hx, lx), 2.0);
    r.mid_y = RN_DIV(RN_ADD(hy, ly), 2.0);
    r.child[0] = r.child[1] = r.child[2] = r.child[3] = STC_NONE;
    bn[0] = r;
    NodeMeta m;
    m.type = NODE_LEAF; m.level = 0; m.overflow = 0; m.underflow = 0; m.grid_id = 0; m.parent = STC_NONE;
    bm[0] = m;
    st->build_nodes = 1;
  }
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) node_of[i] = 0;
}

__global__ void k_build_count(const uint32_t *node_of, uint32_t n, uint32_t a, uint32_t *bcount) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t nid = node_of[i];
  if (nid >= a) atomicAdd(&bcount[nid], 1u);
}

__global__ void k_build_decide(Node *bn, NodeMeta *bm, const uint32_t *bcount, uint32_t a, uint32_t b,
                               uint32_t cap, double reach, uint32_t S, DevState *st) {
  uint32_t nid = a + blockIdx.x * blockDim.x + threadIdx.x;
  if (nid >= b) return;
  Node p = bn[nid];
  bool split = false;
  if (bcount[nid] >= cap) {
    double w = width_geo(p.lo_x, p.lo_y, p.hi_x, RN_MUL(reach, 2.0));
    split = RN_DIV(w, 2.0) > reach;
  }
  if (!split) {
    bm[nid].type = NODE_LEAF;
    return;
  }
  uint32_t c = atomicAdd(&st->build_nodes, 4u);
  if (c + 4 > S) {
    stc_set_error(st, ERR_BUILD, c);
    bm[nid].type = NODE_LEAF;
    return;
  }
  NodeMeta pm = bm[nid];
  for (int i = 0; i < 4; i++) {
    Node ch;
    set_child_box(ch, p, i);
    bn[c + i] = ch;
    NodeMeta m;
    m.type = NODE_LEAF; m.level = (int16_t)(pm.level + 1); m.overflow = 0; m.underflow = 0;
    m.grid_id = 0; m.parent = nid;
    bm[c + i] = m;
    p.child[i] = c + i;
  }
  bn[nid] = p;
  bm[nid].type = NODE_BRANCH;
}

__global__ void k_build_move(const double2 *xy, uint32_t *node_of, uint32_t n, uint32_t a, const Node *bn,
                             const NodeMeta *bm) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t nid = node_of[i];
  if (nid < a || bm[nid].type != NODE_BRANCH) return;
  double2 p = xy[i];
  const Node &q = bn[nid];
  int loc = (p.y > q.mid_y) * 2 + (p.x > q.mid_x);  // QTree.h:191
  node_of[i] = q.child[loc];
}

__global__ void k_build_sub(const Node *bn, const NodeMeta *bm, uint32_t a, uint32_t b, uint32_t *sub_nodes,
                            uint32_t *sub_leaves) {
  uint32_t nid = a + blockIdx.x * blockDim.x + threadIdx.x;
  if (nid >= b) return;
  if (bm[nid].type == NODE_LEAF) {
    sub_nodes[nid] = 1;
    sub_leaves[nid] = 1;
    return;
  }
  uint32_t sn = 1, sl = 0;
  for (int i = 0; i < 4; i++) {
    uint32_t c = bn[nid].child[i];
    sn += sub_nodes[c];
    sl += sub_leaves[c];
  }
  sub_nodes[nid] = sn;
  sub_leaves[nid] = sl;
}

__global__ void k_build_pre_children(const Node *bn, const NodeMeta *bm, uint32_t a, uint32_t b,
                                     const uint32_t *sub_nodes, const uint32_t *sub_leaves, uint32_t *pre,
                                     uint32_t *leafbase) {
  uint32_t nid = a + blockIdx.x * blockDim.x + threadIdx.x;
  if (nid >= b || bm[nid].type != NODE_BRANCH) return;
  uint32_t run = pre[nid] + 1, lb = leafbase[nid];
  for (int i = 0; i < 4; i++) {
    uint32_t c = bn[nid].child[i];
    pre[c] = run;
    leafbase[c] = lb;
    run += sub_nodes[c];
    lb += sub_leaves[c];
  }
}

__global__ void k_build_write(const Node *bn, const NodeMeta *bm, uint32_t total, const uint32_t *pre,
                              const uint32_t *leafbase, SchemaDev sd) {
  uint32_t nid = blockIdx.x * blockDim.x + threadIdx.x;
  if (nid >= total) return;
  uint32_t p = pre[nid];
  Node q = bn[nid];
  NodeMeta m = bm[nid];
  if (m.type == NODE_BRANCH) {
    for (int i = 0; i < 4; i++) q.child[i] = pre[q.child[i]];
    m.grid_id = 0;  // QTNode::node_id of a branch keeps its default 0
  } else {
    m.grid_id = leafbase[nid];
    if (m.grid_id < sd.G) sd.gid_node[m.grid_id] = p;  // overflow is reported by k_build_finish
  }
  m.parent = m.parent == STC_NONE ? STC_NONE : pre[m.parent];
  m.overflow = 0;
  m.underflow = 0;
  sd.nodes[p] = q;
  sd.meta[p] = m;
  sd.fbox[p] = make_float4(__double2float_rn(RN_SUB(q.lo_x, sd.ox)), __double2float_rn(RN_SUB(q.lo_y, sd.oy)),
                           __double2float_rn(RN_SUB(q.hi_x, sd.ox)), __double2float_rn(RN_SUB(q.hi_y, sd.oy)));
}

__global__ void k_build_finish(const uint32_t *sub_nodes, const uint32_t *sub_leaves, uint32_t S, uint32_t G,
                               uint32_t *high, DevState *st) {
  uint32_t nodes = sub_nodes[0], leaves = sub_leaves[0];
  // tracing/filter.cpp:82-85 asserts strict inequality
  if (nodes >= S || leaves >= G) stc_set_error(st, ERR_BUILD, nodes);
  st->schema_stack_index = nodes;
  st->grids_stack_index = leaves;
  high[0] = min(nodes, S);
  high[1] = min(leaves, G);
}

static inline unsigned nblk(size_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

cudaError_t build_schema(const double2 *xy, uint32_t n, const double mbr[4], double reach, uint32_t grid_capacity,
                         SchemaDev sd, SchemaWork w, DevState *st, DevState *st_host, cudaStream_t s) {
  cudaMemsetAsync(sd.meta, 0, (size_t)sd.S * sizeof(NodeMeta), s);
  iota_u32(sd.schema_stack, sd.S, s);
  iota_u32(sd.grids_stack, sd.G, s);
  STC_KL k_build_root<<<nblk(n > 0 ? n : 1), 256, 0, s>>>(w.bnodes, w.bmeta, mbr[0], mbr[1], mbr[2], mbr[3], w.node_of, n,
                                                   st);
  std::vector<uint32_t> ls = {0, 1};
  for (int level = 0; level < STC_MAX_DEPTH; level++) {
    uint32_t a = ls[ls.size() - 2], b = ls.back();
    cudaMemsetAsync(w.bcount + a, 0, (size_t)(b - a) * sizeof(uint32_t), s);
    if (n) STC_KL k_build_count<<<nblk(n), 256, 0, s>>>(w.node_of, n, a, w.bcount);
    STC_KL k_build_decide<<<nblk(b - a), 256, 0, s>>>(w.bnodes, w.bmeta, w.bcount, a, b, grid_capacity, reach, sd.S, st);
    if (n) STC_KL k_build_move<<<nblk(n), 256, 0, s>>>(xy, w.node_of, n, a, w.bnodes, w.bmeta);
    cudaError_t e = cudaMemcpyAsync(st_host, st, sizeof(DevState), cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    if (st_host->error) return cudaSuccess;
    uint32_t total = st_host->build_nodes;
    if (total == b) break;
    ls.push_back(total);
  }
  uint32_t total = ls.back();
  int nlev = (int)ls.size() - 1;
  for (int L = nlev - 1; L >= 0; L--) {
    uint32_t a = ls[L], b = ls[L + 1];
    STC_KL k_build_sub<<<nblk(b - a), 256, 0, s>>>(w.bnodes, w.bmeta, a, b, w.bsub_nodes, w.bsub_leaves);
  }
  cudaMemsetAsync(w.bpre, 0, sizeof(uint32_t), s);  // root: preorder 0, first leaf id 0
  cudaMemsetAsync(w.bleafbase, 0, sizeof(uint32_t), s);
  for (int L = 0; L < nlev; L++) {
    uint32_t a = ls[L], b = ls[L + 1];
    STC_KL k_build_pre_children<<<nblk(b - a), 256, 0, s>>>(w.bnodes, w.bmeta, a, b, w.bsub_nodes, w.bsub_leaves, w.bpre,
                                                     w.bleafbase);
  }
  STC_KL k_build_write<<<nblk(total), 256, 0, s>>>(w.bnodes, w.bmeta, total, w.bpre, w.bleafbase, sd);
  STC_KL k_build_finish<<<1, 1, 0, s>>>(w.bsub_nodes, w.bsub_leaves, sd.S, sd.G, sd.high, st);
  schema_walk(sd, s);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Dynamic update.

enum { EV_NONE = 0, EV_SPLIT = 1, EV_MERGE = 2 };

__global__ void k_schema_phase1(SchemaDev sd, const uint32_t *grid_count, double reach, uint32_t cap, uint32_t delay,
                                uint8_t *ev_flag, int16_t *old_under) {
  const uint32_t high = sd.high[0];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < high; i += gridDim.x * blockDim.x) {
    NodeMeta m = sd.meta[i];
    uint32_t flag = EV_NONE;
    old_under[i] = m.underflow;
    if (m.type == NODE_LEAF) {
      bool cond = false;
      if (grid_count[m.grid_id] > cap) {
        const Node &q = sd.nodes[i];
        double thr = RN_MUL(reach, 2.0);
        cond = width_geo(q.lo_x, q.lo_y, q.hi_x, thr) > thr;
      }
      int16_t nv = cond ? (int16_t)(m.overflow + 1) : (int16_t)0;
      if (cond && (uint32_t)nv >= delay) flag = EV_SPLIT;
      else sd.meta[i].overflow = nv;
    } else if (m.type == NODE_BRANCH) {
      const Node &q = sd.nodes[i];
      int leafchild = 0;
      int ncounter = 0;
      for (int k = 0; k < 4; k++) {
        NodeMeta cm = sd.meta[q.child[k]];
        if (cm.type == NODE_LEAF) {
          leafchild++;
          ncounter += (int)grid_count[cm.grid_id];
        }
      }
      bool cond = leafchild == 4 && (uint32_t)ncounter < cap;
      int16_t nv = cond ? (int16_t)(m.underflow + 1) : (int16_t)0;
      if (cond && (uint32_t)nv >= delay) flag = EV_MERGE;
      else sd.meta[i].underflow = nv;
    }
    ev_flag[i] = (uint8_t)flag;
  }
}

__device__ bool split_node(SchemaDev sd, uint32_t cur, uint32_t *grid_count, DevState *st) {
  // tracing/filter.cpp:338-375
  NodeMeta cm = sd.meta[cur];
  cm.type = NODE_BRANCH;
  if (st->grids_stack_index == 0) return false;
  sd.grids_stack[--st->grids_stack_index] = cm.grid_id;
  Node q = sd.nodes[cur];
  double xhalf = RN_SUB(q.mid_x, q.lo_x);
  double yhalf = RN_SUB(q.mid_y, q.lo_y);
  for (int i = 0; i < 4; i++) {
    if (st->schema_stack_index >= sd.S || st->grids_stack_index >= sd.G) return false;
    uint32_t child = sd.schema_stack[st->schema_stack_index++];
    q.child[i] = child;
    uint32_t g = sd.grids_stack[st->grids_stack_index++];
    grid_count[g] = 0;
    sd.gid_node[g] = child;
    Node c;
    c.lo_x = RN_ADD(q.lo_x, (i % 2 == 1) ? xhalf : 0.0);
    c.lo_y = RN_ADD(q.lo_y, (i / 2 == 1) ? yhalf : 0.0);
    c.hi_x = RN_ADD(q.mid_x, (i % 2 == 1) ? xhalf : 0.0);
    c.hi_y = RN_ADD(q.mid_y, (i / 2 == 1) ? yhalf : 0.0);
    c.mid_x = RN_DIV(RN_ADD(c.lo_x, c.hi_x), 2.0);
    c.mid_y = RN_DIV(RN_ADD(c.lo_y, c.hi_y), 2.0);
    c.child[0] = c.child[1] = c.child[2] = c.child[3] = STC_NONE;
    sd.nodes[child] = c;
    sd.fbox[child] = make_float4(__double2float_rn(RN_SUB(c.lo_x, sd.ox)), __double2float_rn(RN_SUB(c.lo_y, sd.oy)),
                                 __double2float_rn(RN_SUB(c.hi_x, sd.ox)), __double2float_rn(RN_SUB(c.hi_y, sd.oy)));
    NodeMeta m;
    m.type = NODE_LEAF; m.level = (int16_t)(cm.level + 1); m.overflow = 0; m.underflow = 0;
    m.grid_id = g; m.parent = cur;
    sd.meta[child] = m;
  }
  sd.nodes[cur] = q;
  cm.overflow = 0;
  sd.meta[cur] = cm;
  return true;
}

__device__ bool merge_node(SchemaDev sd, uint32_t cur, uint32_t *grid_count, DevState *st) {
  // tracing/filter.cpp:316-336
  Node q = sd.nodes[cur];
  for (int i = 0; i < 4; i++) {
    uint32_t ch = q.child[i];
    NodeMeta m = sd.meta[ch];
    sd.meta[ch].type = NODE_INVALID;
    if (st->schema_stack_index == 0 || st->grids_stack_index == 0) return false;
    sd.schema_stack[--st->schema_stack_index] = ch;
    sd.grids_stack[--st->grids_stack_index] = m.grid_id;
    grid_count[m.grid_id] = 0;
  }
  NodeMeta cm = sd.meta[cur];
  cm.type = NODE_LEAF;
  cm.grid_id = sd.grids_stack[st->grids_stack_index++];
  cm.underflow = 0;
  sd.gid_node[cm.grid_id] = cur;
  sd.meta[cur] = cm;
  return true;
}

// binary min-heap of node indices in global memory (single thread)
__device__ void heap_push(uint32_t *h, uint32_t &n, uint32_t v) {
  uint32_t i = n++;
  h[i] = v;
  while (i > 0) {
    uint32_t p = (i - 1) / 2;
    if (h[p] <= h[i]) break;
    uint32_t t = h[p]; h[p] = h[i]; h[i] = t;
    i = p;
  }
}

__device__ uint32_t heap_pop(uint32_t *h, uint32_t &n) {
  uint32_t top = h[0];
  h[0] = h[--n];
  uint32_t i = 0;
  while (true) {
    uint32_t l = 2 * i + 1, r = l + 1, m = i;
    if (l < n && h[l] < h[m]) m = l;
    if (r < n && h[r] < h[m]) m = r;
    if (m == i) break;
    uint32_t t = h[m]; h[m] = h[i]; h[i] = t;
    i = m;
  }
  return top;
}


// Block replay of the flagged events for the common case: at most
// PAR_MAX_EVENTS events and no merge whose parent has a higher index (the
// only source of a cascade). Without cascades every event's decision is fixed
// by phase 1, and the sequential replay's only coupling is through the two
// free stacks, whose operations have a closed form. A split takes 4 node
// slots off the schema stack and, its own grid id first, 3 more grid ids off
// the grid stack; a merge puts its 4 children's slots and 3 of their grid ids
// back and keeps the fourth. So both stacks move by one group at a time, and
// at level k (splits less merges so far) a split takes group k: what the
// latest earlier merge that ended at level k put there, or the stack's
// content from before the step. Every split looks for its merge among the
// events' levels in shared memory (one thread replaying the stacks took 0.86
// ms of a 10M-object step, which the table update no longer hides; this
// takes 0.03). Node and grid bookkeeping is then written in parallel, merges
// before splits (a node or grid id freed by a merge can only be reused by a
// later split). The per-step grid counts are not reset: nothing reads them
// before the next step recounts.
static constexpr uint32_t PAR_MAX_EVENTS = 4096;

// Per-event scratch in global memory: split -> 4 children, 4 grid ids taken;
// merge -> its 4 children, their 4 grid ids.
struct ParScratch {
  uint32_t *val;  // 8 per event
};

// Largest j < e with v[j] == want, or -1 (v 16-byte aligned).
__device__ __forceinline__ int last_equal(const int *v, int e, int want) {
  int j = e - 1;
  for (; j >= 0 && (j & 3) != 3; j--)
    if (v[j] == want) return j;
  for (; j >= 0; j -= 4) {
    const int4 q = *(const int4 *)&v[j - 3];
    if (q.w == want) return j;
    if (q.z == want) return j - 1;
    if (q.y == want) return j - 2;
    if (q.x == want) return j - 3;
  }
  return -1;
}

// Block-wide exclusive scan of one value per thread of a 1024-thread block;
// total receives the sum. warp_sum: 32 words of shared memory.
__device__ __forceinline__ int block_scan(int v, int *warp_sum, int &total) {
  const uint32_t lane = threadIdx.x & 31u;
  int incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, d);
    if ((int)lane >= d) incl += up;
  }
  __syncthreads();  // the last use of warp_sum is over
  if (lane == 31) warp_sum[threadIdx.x >> 5] = incl;
  __syncthreads();
  int before = incl - v;
  total = 0;
  for (uint32_t w = 0; w < 32; w++) {
    if (w < (threadIdx.x >> 5)) before += warp_sum[w];
    total += warp_sum[w];
  }
  return before;
}

// The whole block; false when the events need the one-thread replay.
__device__ __forceinline__ bool replay_block(const SchemaDev &sd, const uint32_t *ev_list, uint32_t nev,
                                             uint32_t *scratch, DevState *st, int *warp_sum) {
  __shared__ uint32_t sh_node[PAR_MAX_EVENTS];
  __shared__ __align__(16) int sh_lev[PAR_MAX_EVENTS];  // 4 * (level before the event) + kind
  __shared__ int cascade, bad;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) cascade = bad = 0;
  if (nev > PAR_MAX_EVENTS) return false;
  ParScratch ps{scratch};
  const int ssi0 = (int)st->schema_stack_index, gsi0 = (int)st->grids_stack_index;
  __syncthreads();
  // thread t owns events [t * per, (t + 1) * per)
  const uint32_t per = (nev + blockDim.x - 1) / blockDim.x, e0 = min(tid * per, nev), e1 = min(e0 + per, nev);
  int sum = 0;
  for (uint32_t e = e0; e < e1; e++) {
    const uint32_t v = ev_list[e], node = v >> 2, kind = v & 3u;
    sh_node[e] = node;
    sh_lev[e] = (int)kind;
    sum += kind == EV_SPLIT ? 1 : -1;
    if (kind == EV_MERGE) {
      uint32_t par = sd.meta[node].parent;
      if (node != 0 && par != STC_NONE && par > node) cascade = 1;
      Node q = sd.nodes[node];
      for (int i = 0; i < 4; i++) {
        ps.val[8 * e + i] = q.child[i];
        ps.val[8 * e + 4 + i] = sd.meta[q.child[i]].grid_id;
      }
    } else {
      ps.val[8 * e + 4] = sd.meta[node].grid_id;  // the split's own grid id goes to its first child
    }
  }
  int total = 0;
  int level = block_scan(sum, warp_sum, total);
  if (cascade) return false;
  for (uint32_t e = e0; e < e1; e++) {
    const int kind = sh_lev[e], si = ssi0 + 4 * level, gi = gsi0 + 3 * level;
    sh_lev[e] = level * 4 + kind;
    if (kind == EV_SPLIT) {
      if (si + 4 > (int)sd.S || gi - 1 < 0 || gi + 3 > (int)sd.G) bad = 1;
      level++;
    } else {
      if (si - 4 < 0 || gi - 4 < 0) bad = 1;
      level--;
    }
  }
  __syncthreads();
  if (bad) {
    if (tid == 0) stc_set_error(st, ERR_SCHEMA, 0u);
    return true;
  }
  for (uint32_t e = tid; e < nev; e += blockDim.x) {
    const int lk = sh_lev[e], k = lk >> 2;
    uint32_t *v = ps.val + 8 * e;
    if ((lk & 3) == EV_SPLIT) {
      // the latest earlier merge from level k + 1
      const int j = last_equal(sh_lev, (int)e, (k + 1) * 4 + EV_MERGE);
      if (j >= 0) {
        const uint32_t *m = ps.val + 8 * j;
        for (int i = 0; i < 4; i++) v[i] = m[3 - i];
        for (int i = 1; i < 4; i++) v[4 + i] = m[4 + 3 - i];
      } else {
        for (int i = 0; i < 4; i++) v[i] = sd.schema_stack[ssi0 + 4 * k + i];
        for (int i = 1; i < 4; i++) v[4 + i] = sd.grids_stack[gsi0 + 3 * k + i - 1];
      }
    }
  }
  __syncthreads();
  // what the step leaves on the stacks: each free group's last merge
  for (uint32_t e = tid; e < nev; e += blockDim.x) {
    const int lk = sh_lev[e], k = (lk >> 2) - 1;  // the group a merge fills
    if ((lk & 3) != EV_MERGE || k < total) continue;
    uint32_t j = e + 1;
    while (j < nev && sh_lev[j] != lk) j++;
    if (j < nev) continue;  // filled again later
    const uint32_t *m = ps.val + 8 * e;
    for (int i = 0; i < 4; i++) sd.schema_stack[ssi0 + 4 * k + 3 - i] = m[i];
    for (int i = 0; i < 3; i++) sd.grids_stack[gsi0 + 3 * k + 2 - i] = m[4 + i];
  }
  if (tid == 0) {
    st->schema_stack_index = (uint32_t)(ssi0 + 4 * total);
    st->grids_stack_index = (uint32_t)(gsi0 + 3 * total);
  }
  // merges (tracing/filter.cpp:316-336)
  for (uint32_t e = tid; e < nev; e += blockDim.x) {
    if ((sh_lev[e] & 3) != EV_MERGE) continue;
    uint32_t cur = sh_node[e];
    const uint32_t *v = ps.val + 8 * e;
    for (int i = 0; i < 4; i++) sd.meta[v[i]].type = NODE_INVALID;
    NodeMeta cm = sd.meta[cur];
    cm.type = NODE_LEAF;
    cm.grid_id = v[7];  // the pop returns the last pushed grid id
    cm.underflow = 0;
    sd.meta[cur] = cm;
    sd.gid_node[v[7]] = cur;
  }
  __syncthreads();
  // splits (tracing/filter.cpp:338-375)
  for (uint32_t e = tid; e < nev; e += blockDim.x) {
    if ((sh_lev[e] & 3) != EV_SPLIT) continue;
    uint32_t cur = sh_node[e];
    const uint32_t *v = ps.val + 8 * e;
    Node q = sd.nodes[cur];
    NodeMeta cm = sd.meta[cur];
    double xhalf = RN_SUB(q.mid_x, q.lo_x);
    double yhalf = RN_SUB(q.mid_y, q.lo_y);
    for (int i = 0; i < 4; i++) {
      uint32_t child = v[i], gid = v[4 + i];
      Node c;
      c.lo_x = RN_ADD(q.lo_x, (i % 2 == 1) ? xhalf : 0.0);
      c.lo_y = RN_ADD(q.lo_y, (i / 2 == 1) ? yhalf : 0.0);
      c.hi_x = RN_ADD(q.mid_x, (i % 2 == 1) ? xhalf : 0.0);
      c.hi_y = RN_ADD(q.mid_y, (i / 2 == 1) ? yhalf : 0.0);
      c.mid_x = RN_DIV(RN_ADD(c.lo_x, c.hi_x), 2.0);
      c.mid_y = RN_DIV(RN_ADD(c.lo_y, c.hi_y), 2.0);
      c.child[0] = c.child[1] = c.child[2] = c.child[3] = STC_NONE;
      sd.nodes[child] = c;
      sd.fbox[child] = make_float4(__double2float_rn(RN_SUB(c.lo_x, sd.ox)), __double2float_rn(RN_SUB(c.lo_y, sd.oy)),
                                   __double2float_rn(RN_SUB(c.hi_x, sd.ox)), __double2float_rn(RN_SUB(c.hi_y, sd.oy)));
      NodeMeta m;
      m.type = NODE_LEAF; m.level = (int16_t)(cm.level + 1); m.overflow = 0; m.underflow = 0;
      m.grid_id = gid; m.parent = cur;
      sd.meta[child] = m;
      sd.gid_node[gid] = child;
      q.child[i] = child;
    }
    sd.nodes[cur] = q;
    cm.type = NODE_BRANCH;
    cm.overflow = 0;
    sd.meta[cur] = cm;
  }
  __syncthreads();
  if (tid == 0) {
    st->splits = (uint32_t)((int)nev + total) / 2;
    st->merges = (uint32_t)((int)nev - total) / 2;
  }
  return true;
}

// One thread, in the reference's order, with cascades.
__device__ void replay_serial(const SchemaDev &sd, uint32_t *grid_count, const uint32_t *ev_list, uint32_t nev,
                              const int16_t *old_under, uint32_t *heap, uint8_t *queued, uint32_t cap, uint32_t delay,
                              DevState *st) {
  uint32_t hn = 0, ei = 0;
  uint32_t splits = 0, merges = 0;
  while (ei < nev || hn > 0) {
    uint32_t ev_node = ei < nev ? (ev_list[ei] >> 2) : 0xFFFFFFFFu;
    uint32_t h_node = hn > 0 ? heap[0] : 0xFFFFFFFFu;
    if (h_node < ev_node) {
      uint32_t p = heap_pop(heap, hn);
      queued[p] = 0;
      // re-evaluate the branch rule at p's own visit (filter.cpp:399-420)
      NodeMeta pm = sd.meta[p];
      if (pm.type != NODE_BRANCH) continue;
      const Node &q = sd.nodes[p];
      int leafchild = 0, ncounter = 0;
      for (int k = 0; k < 4; k++) {
        NodeMeta cm = sd.meta[q.child[k]];
        if (cm.type == NODE_LEAF) {
          leafchild++;
          ncounter += (int)grid_count[cm.grid_id];
        }
      }
      bool cond = leafchild == 4 && (uint32_t)ncounter < cap;
      int16_t nv = cond ? (int16_t)(old_under[p] + 1) : (int16_t)0;
      if (cond && (uint32_t)nv >= delay) {
        if (!merge_node(sd, p, grid_count, st)) { stc_set_error(st, ERR_SCHEMA, p); return; }
        merges++;
        uint32_t pp = sd.meta[p].parent;
        if (p != 0 && pp != STC_NONE && pp > p && !queued[pp]) { queued[pp] = 1; heap_push(heap, hn, pp); }
      } else {
        sd.meta[p].underflow = nv;
      }
      continue;
    }
    if (h_node == ev_node) {  // an event node is never a pending parent; drop the duplicate
      heap_pop(heap, hn);
      queued[h_node] = 0;
    }
    uint32_t e = ev_list[ei++];
    uint32_t node = e >> 2, kind = e & 3u;
    if (kind == EV_SPLIT) {
      if (!split_node(sd, node, grid_count, st)) { stc_set_error(st, ERR_SCHEMA, node); return; }
      splits++;
    } else {
      if (!merge_node(sd, node, grid_count, st)) { stc_set_error(st, ERR_SCHEMA, node); return; }
      merges++;
      uint32_t pp = sd.meta[node].parent;
      if (node != 0 && pp != STC_NONE && pp > node && !queued[pp]) { queued[pp] = 1; heap_push(heap, hn, pp); }
    }
  }
  st->splits = splits;
  st->merges = merges;
}

// The flagged nodes in index order, then their replay. One block: thread t
// collects the flags of nodes [t * per, (t + 1) * per).
__global__ void __launch_bounds__(1024) k_schema_phase2(SchemaDev sd, SchemaWork w, uint32_t *grid_count, uint32_t cap,
                                                        uint32_t delay, int serial_only, DevState *st) {
  after_previous();
  __shared__ int warp_sum[32];
  const uint32_t tid = threadIdx.x, high = sd.high[0];
  const uint32_t per = ((high + 1023) / 1024 + 15) / 16 * 16;
  const uint32_t n0 = min(tid * per, high), n1 = min(n0 + per, high);
  int count = 0;
  for (uint32_t i = n0; i < n1; i += 16) {
    const uint4 f = *(const uint4 *)&w.ev_flag[i];  // flags past the last node are 0
    const uint32_t v[4] = {f.x, f.y, f.z, f.w};
    for (int k = 0; k < 4; k++) count += __popc((v[k] | v[k] >> 1) & 0x01010101u);
  }
  int total = 0;
  int at = block_scan(count, warp_sum, total);
  if (count)
    for (uint32_t i = n0; i < n1; i++) {
      const uint32_t f = w.ev_flag[i];
      if (f) w.ev_list[at++] = i << 2 | f;
    }
  __syncthreads();
  const uint32_t ssi0 = st->schema_stack_index, gsi0 = st->grids_stack_index;
  __syncthreads();
  uint32_t path = 0;
  if (!serial_only) path = replay_block(sd, w.ev_list, (uint32_t)total, w.par_scratch, st, warp_sum) ? 1u : 2u;
  if (tid) return;
  if (path != 1) replay_serial(sd, grid_count, w.ev_list, (uint32_t)total, w.old_under, w.heap, w.queued, cap, delay, st);
  st->schema_path = path;
  // ids ever handed out: a split takes at most 4 node and 3 more grid ids
  sd.high[0] = min(max(high, ssi0 + 4 * st->splits), sd.S);
  sd.high[1] = min(max(sd.high[1], gsi0 + 3 * st->splits), sd.G);
}

__global__ void __launch_bounds__(256) k_schema_walk(SchemaDev sd) {
  after_previous();
  const uint32_t high = sd.high[0];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < high; i += gridDim.x * blockDim.x) {
    const NodeMeta m = sd.meta[i];
    if (i == 0) sd.start[sd.start_edge * sd.start_edge] = m.type == NODE_LEAF ? (m.grid_id | WALK_LEAF) : 0u;
    if (m.type != NODE_BRANCH) continue;
    const Node *n = &sd.nodes[i];
    const uint4 c = *(const uint4 *)n->child;
    uint32_t ch[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const NodeMeta cm = sd.meta[ch[k]];
      // (an invalid child stands for no node: the descent reports it)
      if (cm.type == NODE_LEAF) ch[k] = cm.grid_id | WALK_LEAF;
      else if (cm.type != NODE_BRANCH) ch[k] = STC_NONE;
    }
    Walk w;
    w.mid_x = order_key(__double_as_longlong(n->mid_x));
    w.mid_y = order_key(__double_as_longlong(n->mid_y));
    for (int k = 0; k < 4; k++) w.child[k] = ch[k];
    sd.walk[i] = w;
    const float4 b = sd.fbox[i];
    sd.wbox[i] = WalkBox{b.x, b.y, b.z, b.w, __double2float_rn(RN_SUB(n->mid_x, sd.ox)),
                         __double2float_rn(RN_SUB(n->mid_y, sd.oy)), {0.f, 0.f}};
  }
}

// A cell's corners, widened by 2e-3 of it and dozens of the coordinates' last
// places (several times the rounding of a point's float cell number, at most
// 1024 cells times a few 2^-24), walk down together while they take the same
// child: the descent compares each coordinate with the split points alone, so
// every point between them takes it too.
__global__ void __launch_bounds__(256) k_schema_start(SchemaDev sd) {
  after_previous();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, E = sd.start_edge;
  if (i >= E * E) return;
  const double cx = 1.0 / (double)sd.start_sx, cy = 1.0 / (double)sd.start_sy;
  const double ix = (double)(i % E), iy = (double)(i / E);
  const double wx = 2e-3 * cx + 1e-14 * (fabs(sd.ox) + E * cx), wy = 2e-3 * cy + 1e-14 * (fabs(sd.oy) + E * cy);
  const double x0 = sd.ox + ix * cx - wx, x1 = sd.ox + (ix + 1.0) * cx + wx;
  const double y0 = sd.oy + iy * cy - wy, y1 = sd.oy + (iy + 1.0) * cy + wy;
  uint32_t cur = sd.start[E * E];
  for (int d = 0; !(cur & WALK_LEAF) && d < STC_MAX_DEPTH; d++) {
    const double mx = sd.nodes[cur].mid_x, my = sd.nodes[cur].mid_y;
    if ((x0 > mx) != (x1 > mx) || (y0 > my) != (y1 > my)) break;
    cur = sd.walk[cur].child[(y0 > my) * 2 + (x0 > mx)];
  }
  sd.start[i] = cur;
}

void schema_walk(SchemaDev sd, cudaStream_t s) {
  launch_behind(k_schema_walk, std::min<unsigned>(nblk(sd.S), num_sms() * 4), 256, 0, s, sd);
  launch_behind(k_schema_start, nblk((size_t)sd.start_edge * sd.start_edge), 256, 0, s, sd);
}

void update_schema(SchemaDev sd, SchemaWork w, uint32_t *grid_count, double reach, uint32_t grid_capacity,
                   uint32_t delay, int serial_only, DevState *st, cudaStream_t s) {
  STC_KL k_schema_phase1<<<std::min<unsigned>(nblk(sd.S), num_sms() * 4), 256, 0, s>>>(
      sd, grid_count, reach, grid_capacity, delay, w.ev_flag, w.old_under);
  launch_behind(k_schema_phase2, 1, 1024, 0, s, sd, w, grid_count, grid_capacity, delay, serial_only, st);
  schema_walk(sd, s);
}

}  // namespace stc
