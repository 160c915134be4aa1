// Work lists of the outgoing plane-wave pass and the tree's box lists, laid
// out on the device (plan.cu).
#pragma once
#include <cuda_runtime.h>

#include "tree.hpp"

namespace pdmk {

// One box, or one split-K chunk of a box, of the outgoing pass over a range
// of the particles in leaf order (rows x, y, z, q without the leaves' free
// slots, which were 26 % of the slots at N = 1e6). `tab`: the chunk tables
// of the range (mixed pass only).
struct PwItem {
  double cx, cy, cz;  // box centre
  double dk;          // mode spacing of the box's level
  int X, Y, Z;        // integer box coordinates at its level
  int M;              // decentring multiplier: 1 for levels >= 2, 3 for the root
  int s_begin, s_end;
  double2* out;        // the box's H complex outputs (or its split-K partial)
  unsigned char* tab;
};

// A box summed from n split-K partials, the first of them at row `first`.
struct PwSplit {
  int first, n;
  double2* out;
};

// Totals of the tree's lists: read back once, they size the buffers.
constexpr int kPlanBuckets = 128;  // box sizes, four buckets per octave
struct PlanTotals {
  int n_items, n_chunks, n_split, n_split_items;
  int n_nonleaf, n_leaves, n_cubes, pad;
};
struct PlanState {
  PlanTotals t;
  int hist[kPlanBuckets];    // items per size bucket
  int cursor[kPlanBuckets];  // items placed so far
  int cur_chunk, cur_split, cur_split_item, pad;
};

// Split of the particle ranges: boxes above ksplit particles are cut into
// items of ksplit; kcp particles per table chunk of tab_bytes (mixed; 0: no tables)
struct PlanShape {
  int ksplit, kcp;
  long tab_bytes;
};

int plan_blocks(int n_nodes);
// the root's items, chunk list and split entry (grid-sized by the host); *next = 0
void launch_plan_root(const DevTree& T, const PlanShape& s, int n, int n_items, int n_chunks, double2* part,
                      unsigned char* tab, PwItem* items, int2* chunks, PwSplit* split, int* next, cudaStream_t st);
// totals over the nodes into *state (zeroed by the caller); `lists`: the box
// lists' as well, with per-block counts in blk[3 plan_blocks]
void launch_plan_count(const DevTree& T, const PlanShape& s, bool lists, PlanState* state, int* blk, cudaStream_t st);
// the box lists in node order
void launch_plan_lists(const DevTree& T, const int* blk, int* nonleaf, int* leaves, int* cubes, cudaStream_t st);
// the items in order of falling size, their chunk list and the split boxes;
// *next = 0
void launch_plan_items(const DevTree& T, const PlanShape& s, const int* node_first, PlanState* state, double2* part,
                       unsigned char* tab, PwItem* items, int2* chunks, PwSplit* split, int* next, cudaStream_t st);

}  // namespace pdmk
