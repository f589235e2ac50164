// Quadtree schema on the device: build at create, dynamic update per step.
#pragma once
#include "stc_common.cuh"

namespace stc {

// FP64 runs at 2 lanes a clock here (a warp's compare or conversion takes as
// long as 64 of its FP32 instructions on four issue slots), so the step's
// per-object walks compare coordinates as integers and as bounded floats.

// A branch as the descent reads it, in one 32-byte load: its split point as
// order keys (order_key) and its children, a leaf as WALK_LEAF | grid id.
// WalkBox: its box and split point in float degrees from the map's corner.
// Rebuilt from nodes and meta after every schema change (schema_walk).
#define WALK_LEAF 0x80000000u
struct __align__(32) Walk {
  long long mid_x, mid_y;
  uint32_t child[4];
};
struct __align__(32) WalkBox {
  float lo_x, lo_y, hi_x, hi_y, mid_x, mid_y, pad[2];
};

// Integers in the order of the doubles (both zeros alike); NaN below all, so
// that it is greater than no split point, as in the comparison of doubles.
__host__ __device__ __forceinline__ long long order_key(long long bits) {
  const unsigned long long mag = (unsigned long long)bits & 0x7FFFFFFFFFFFFFFFull;
  if (mag > 0x7FF0000000000000ull) return (long long)0x8000000000000000ull;
  return bits < 0 ? -(long long)mag : bits;
}

struct SchemaDev {
  Node *nodes;            // S
  Walk *walk;             // S; valid for branches
  WalkBox *wbox;          // S; valid for branches
  // Where descents start: the map cut into start_edge x start_edge cells, and
  // for each the deepest node every point of the cell (a little widened)
  // passes through, as a child word. Points outside the map start at the
  // root (the entry behind the cells).
  uint32_t *start;        // start_edge^2 + 1
  uint32_t start_edge;
  float start_sx, start_sy;  // cells per degree
  NodeMeta *meta;         // S
  uint32_t *schema_stack; // S
  uint32_t *grids_stack;  // G
  uint32_t *gid_node;     // G: leaf grid id -> node index
  float4 *fbox;           // S: node box in fp32 degrees relative to (ox, oy)
  double ox, oy;          // map origin for fbox
  uint32_t *high;         // 2: node ids and grid ids ever handed out lie below these
  uint32_t S, G;
};

struct SchemaWork {
  // build temporaries
  Node *bnodes;
  NodeMeta *bmeta;
  uint32_t *bcount, *bsub_nodes, *bsub_leaves, *bpre, *bleafbase;
  uint32_t *node_of;      // N
  // update temporaries
  uint8_t *ev_flag;       // S, padded with zeros to a multiple of 16 (0 none, 1 split, 2 merge)
  uint32_t *ev_list;      // S
  int16_t *old_under;     // S
  uint32_t *heap;         // S
  uint8_t *queued;        // S
  uint32_t *par_scratch;  // 8 * 4096 words for the block replay
};

// Builds the schema from step-0 positions (index/QTree.h:157-311 semantics:
// a node splits iff at least grid_capacity points descend into it and its
// geographic width / 2 exceeds reach). Returns cudaSuccess or an error; on a
// capacity problem sets st->error = ERR_BUILD.
cudaError_t build_schema(const double2 *xy, uint32_t n, const double mbr[4], double reach,
                         uint32_t grid_capacity, SchemaDev sd, SchemaWork w, DevState *st, DevState *st_host,
                         cudaStream_t s);

// Dynamic update after a step (tracing/filter.cpp:377-449).
// serial_only forces the one-thread replay (the parallel one is used when it applies).
// Rebuilds walk and start.
void schema_walk(SchemaDev sd, cudaStream_t s);
void update_schema(SchemaDev sd, SchemaWork w, uint32_t *grid_count, double reach, uint32_t grid_capacity,
                   uint32_t delay, int serial_only, DevState *st, cudaStream_t s);

}  // namespace stc
