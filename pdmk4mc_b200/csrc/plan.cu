// Work lists of the outgoing plane-wave pass (form_outgoing_pw,
// src/planewave.cpp:31-97) and the tree's box lists, laid out on the device.
//
// A host layout read the nodes back (20 bytes each), sorted the boxes and
// wrote one item per 128-row tile: 1.0 ms at N = 1e6 and 8 ms on a clustered
// tree of 8e4 nodes at 12 digits, during which the device held only the root
// pass. Here a count pass, one read-back of 32 bytes for the buffer sizes
// and a fill pass take its place.
#include <algorithm>

#include "common.cuh"
#include "plan.hpp"

namespace pdmk {

namespace {

constexpr int PLAN_T = 256;  // nodes of a block

// Size bucket of a box: four per octave, the largest boxes first. The order
// only sets which blocks start first (a long item that starts last would run
// on alone), so a quarter octave is fine enough.
__device__ __forceinline__ int size_bucket(int n) {
  if (n <= 0) return kPlanBuckets - 1;
  const int b = int(__float_as_uint(float(n)) >> 21) - (127 << 2);
  return max(0, kPlanBuckets - 1 - b);
}

__device__ __forceinline__ int items_of(const PlanShape& s, int n) {
  return n > s.ksplit ? (n + s.ksplit - 1) / s.ksplit : 1;
}
__device__ __forceinline__ int chunks_of(const PlanShape& s, int n) {
  if (s.tab_bytes == 0) return 0;
  const int full = (s.ksplit + s.kcp - 1) / s.kcp, k = items_of(s, n);
  return (k - 1) * full + (n - (k - 1) * s.ksplit + s.kcp - 1) / s.kcp;
}

__device__ __forceinline__ bool has_expansion(const DevTree& T, int id) {
  return T.pw_hi >= T.pw_lo && id >= T.level_start[T.pw_lo] && id < T.level_start_d[T.pw_hi + 1];
}

// what the box lists say of a node: 1 non-leaf of an expansion level, 2 leaf
// at levels >= 2, 4 box two levels above the expansion levels with a non-leaf
// grandchild (it names the 4 x 4 x 4 receivers of one incoming block)
__device__ __forceinline__ int list_flags(const DevTree& T, int id) {
  const int c = T.node_child0[id];
  int f = 0;
  if (c < 0) {
    if (id >= T.level_start[2]) f |= 2;
    return f;
  }
  if (has_expansion(T, id)) f |= 1;
  if (T.pw_hi >= T.pw_lo && id >= T.level_start_d[T.pw_lo - 2] && id < T.level_start_d[T.pw_hi - 1]) {
    bool any = false;
    for (int a = 0; a < 8 && !any; ++a) {
      const int ch = T.node_child0[c + a];
      if (ch < 0) continue;
      for (int b = 0; b < 8; ++b) any = any || T.node_child0[ch + b] >= 0;
    }
    if (any) f |= 4;
  }
  return f;
}

__device__ __forceinline__ PwItem box_item(const DevTree& T, int l, uint64_t p, double dk, int sb, int se) {
  PwItem w;
  const double scale = ldexp(1.0, -l);
  w.X = int(compact3(p));
  w.Y = int(compact3(p >> 1));
  w.Z = int(compact3(p >> 2));
  // X scale + scale / 2 is exact
  w.cx = T.L * (double(w.X) * scale + 0.5 * scale);
  w.cy = T.L * (double(w.Y) * scale + 0.5 * scale);
  w.cz = T.L * (double(w.Z) * scale + 0.5 * scale);
  w.dk = dk;
  w.M = l == 0 ? 3 : 1;
  w.s_begin = sb;
  w.s_end = se;
  w.out = nullptr;
  w.tab = nullptr;
  return w;
}

__global__ void k_plan_root(DevTree T, PlanShape s, int n, int n_items, int n_chunks, double dk, double2* part,
                            unsigned char* tab, PwItem* items, int2* chunks, PwSplit* split, int* next) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int full = s.tab_bytes ? (s.ksplit + s.kcp - 1) / s.kcp : 1;
  if (i < n_items) {
    PwItem w = box_item(T, 0, 0, dk, i * s.ksplit, min(n, (i + 1) * s.ksplit));
    w.out = part + size_t(i) * T.Hw;
    w.tab = tab + size_t(i) * full * s.tab_bytes;
    items[i] = w;
  }
  if (i < n_chunks) chunks[i] = make_int2(i / full, i % full);
  if (i == 0) {
    *split = PwSplit{0, n_items, T.out_root};
    *next = 0;
  }
}

__global__ void k_plan_count(DevTree T, PlanShape s, bool lists, PlanState* state, int* blk) {
  __shared__ int hist[kPlanBuckets];
  __shared__ int sum[4];
  const int id = blockIdx.x * PLAN_T + threadIdx.x;
  for (int i = threadIdx.x; i < kPlanBuckets; i += PLAN_T) hist[i] = 0;
  if (threadIdx.x < 4) sum[threadIdx.x] = 0;
  __syncthreads();
  const bool in = id < T.n_nodes;
  if (in && has_expansion(T, id)) {
    const int n = T.node_count[id], k = items_of(s, n);
    atomicAdd(&hist[size_bucket(n)], k);
    atomicAdd(&sum[0], k);
    const int c = chunks_of(s, n);
    if (c) atomicAdd(&sum[1], c);
    if (k > 1) {
      atomicAdd(&sum[2], 1);
      atomicAdd(&sum[3], k);
    }
  }
  const int f = in && lists ? list_flags(T, id) : 0;
  const int n0 = __syncthreads_count(f & 1), n1 = __syncthreads_count(f & 2), n2 = __syncthreads_count(f & 4);
  for (int i = threadIdx.x; i < kPlanBuckets; i += PLAN_T)
    if (hist[i]) atomicAdd(&state->hist[i], hist[i]);
  if (threadIdx.x < 4 && sum[threadIdx.x]) atomicAdd(&state->t.n_items + threadIdx.x, sum[threadIdx.x]);
  if (lists && threadIdx.x < 3) {
    const int v = threadIdx.x == 0 ? n0 : threadIdx.x == 1 ? n1 : n2;
    blk[threadIdx.x * gridDim.x + blockIdx.x] = v;
    if (v) atomicAdd(&state->t.n_nonleaf + threadIdx.x, v);
  }
}

// Compaction in node order (the energy sums run over these lists, so their
// order is part of the result): a block adds up the counts of the blocks
// before it, at most a few hundred.
__global__ void __launch_bounds__(PLAN_T) k_plan_lists(DevTree T, const int* __restrict__ blk, int* nonleaf,
                                                       int* leaves, int* cubes) {
  __shared__ int base[3], wcnt[3][PLAN_T / 32];
  if (threadIdx.x < 3) base[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    int v = 0;
    for (int b = threadIdx.x; b < int(blockIdx.x); b += PLAN_T) v += blk[j * gridDim.x + b];
    if (v) atomicAdd(&base[j], v);
  }
  const int id = blockIdx.x * PLAN_T + threadIdx.x;
  const int f = id < T.n_nodes ? list_flags(T, id) : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned m[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    m[j] = __ballot_sync(~0u, (f >> j) & 1);
    if (lane == 0) wcnt[j][warp] = __popc(m[j]);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    if (!((f >> j) & 1)) continue;
    int p = base[j] + __popc(m[j] & ((1u << lane) - 1));
    for (int w = 0; w < warp; ++w) p += wcnt[j][w];
    (j == 0 ? nonleaf : j == 1 ? leaves : cubes)[p] = id;
  }
}

__global__ void __launch_bounds__(PLAN_T)
    k_plan_items(DevTree T, PlanShape s, const int* __restrict__ node_first, PlanState* state, double2* part,
                 unsigned char* tab, PwItem* items, int2* chunks, PwSplit* split, int* next) {
  __shared__ int start[kPlanBuckets], cnt[kPlanBuckets];
  __shared__ int n_ch, ch0;
  for (int i = threadIdx.x; i < kPlanBuckets; i += PLAN_T) cnt[i] = 0;
  if (threadIdx.x == 0) n_ch = 0;
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    *next = 0;
    // every outgoing row is about to be written: the pass has all its memory (had
    // it failed, a later call would find the rows undefined and clear them)
    T.counter[14] = 1;
  }
  // exclusive sums of the buckets: four per lane of the first warp
  if (threadIdx.x < 32) {
    int h[4], v = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      h[i] = v;
      v += state->hist[threadIdx.x * 4 + i];
    }
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(~0u, inc, o);
      if (int(threadIdx.x) >= o) inc += u;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) start[threadIdx.x * 4 + i] = inc - v + h[i];
  }
  __syncthreads();
  const int id = T.level_start[T.pw_lo] + blockIdx.x * PLAN_T + threadIdx.x;
  const bool in = id < T.n_nodes && has_expansion(T, id);
  const int n = in ? T.node_count[id] : 0;
  const int k = items_of(s, n), nc = in ? chunks_of(s, n) : 0;
  const int bu = size_bucket(n);
  int pos = 0, cpos = 0;
  if (in) {
    pos = atomicAdd(&cnt[bu], k);
    if (nc) cpos = atomicAdd(&n_ch, nc);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kPlanBuckets; i += PLAN_T)
    if (cnt[i]) start[i] += atomicAdd(&state->cursor[i], cnt[i]);
  if (threadIdx.x == 0) ch0 = n_ch ? atomicAdd(&state->cur_chunk, n_ch) : 0;
  __syncthreads();
  if (!in) return;
  pos += start[bu];
  cpos += ch0;
  const int l = T.node_level[id];
  const int sb = node_first[id];
  double2* out = T.out + size_t(id - T.pw_base) * T.H;
  if (k > 1) {
    const int first = atomicAdd(&state->cur_split_item, k);
    split[atomicAdd(&state->cur_split, 1)] = PwSplit{first, k, out};
    out = part + size_t(first) * T.H;
  }
  const PwItem w0 = box_item(T, l, T.node_prefix[id], level_dk(T, l), sb, sb + n);
  for (int c = 0; c < k; ++c) {
    PwItem w = w0;
    w.s_begin = sb + c * s.ksplit;
    w.s_end = c + 1 < k ? w.s_begin + s.ksplit : sb + n;
    w.out = out + size_t(c) * T.H;
    w.tab = tab + size_t(cpos) * s.tab_bytes;
    items[pos + c] = w;
    if (s.tab_bytes) {
      const int m = (w.s_end - w.s_begin + s.kcp - 1) / s.kcp;
      for (int q = 0; q < m; ++q) chunks[cpos + q] = make_int2(pos + c, q);
      cpos += m;
    }
  }
}

}  // namespace

int plan_blocks(int n_nodes) { return (n_nodes + PLAN_T - 1) / PLAN_T; }

void launch_plan_root(const DevTree& T, const PlanShape& s, int n, int n_items, int n_chunks, double2* part,
                      unsigned char* tab, PwItem* items, int2* chunks, PwSplit* split, int* next,
                       cudaStream_t st) {
  const int m = std::max(n_items, n_chunks);
  k_plan_root<<<unsigned((m + 127) / 128), 128, 0, st>>>(T, s, n, n_items, n_chunks, T.delta_k[0], part, tab, items,
                                                         chunks, split, next);
  PDMK_LAUNCH_CHECK();
}

void launch_plan_count(const DevTree& T, const PlanShape& s, bool lists, PlanState* state, int* blk, cudaStream_t st) {
  k_plan_count<<<unsigned(plan_blocks(T.n_nodes)), PLAN_T, 0, st>>>(T, s, lists, state, blk);
  PDMK_LAUNCH_CHECK();
}

void launch_plan_lists(const DevTree& T, const int* blk, int* nonleaf, int* leaves, int* cubes, cudaStream_t st) {
  k_plan_lists<<<unsigned(plan_blocks(T.n_nodes)), PLAN_T, 0, st>>>(T, blk, nonleaf, leaves, cubes);
  PDMK_LAUNCH_CHECK();
}

void launch_plan_items(const DevTree& T, const PlanShape& s, const int* node_first, PlanState* state, double2* part,
                       unsigned char* tab, PwItem* items, int2* chunks, PwSplit* split, int* next,
                       cudaStream_t st) {
  if (T.pw_hi < T.pw_lo) return;
  const int n_pw = T.level_start[T.pw_hi + 1] - T.level_start[T.pw_lo];
  if (n_pw == 0) return;
  k_plan_items<<<unsigned(plan_blocks(n_pw)), PLAN_T, 0, st>>>(T, s, node_first, state, part, tab, items, chunks,
                                                              split, next);
  PDMK_LAUNCH_CHECK();
}

}  // namespace pdmk
