// Exclusive scan (one launch up to 4096 items, else reduce-then-scan in three
// launches) and stable LSD radix sort with 8-bit digits (one histogram launch
// for all digits, then one launch a digit: stable warp-multisplit ranks, each
// tile's place from its predecessors' published counts). Used to bin particles
// by Morton key.
#include <algorithm>

#include "common.cuh"
#include "sort.cuh"

namespace pdmk {
namespace {

constexpr int SCAN_T = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_T * SCAN_ITEMS;

__device__ inline int block_exclusive_scan_1024(int v, int* smem32, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem32[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < (blockDim.x >> 5) ? smem32[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    smem32[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  int warp_off = warp > 0 ? smem32[warp - 1] : 0;
  if (total) *total = smem32[(blockDim.x >> 5) - 1];
  return warp_off + x - v;
}

__global__ void k_block_sums(const int* in, long n, int* bsum) {
  long base = long(blockIdx.x) * SCAN_TILE;
  int s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    long i = base + long(threadIdx.x) * SCAN_ITEMS + k;
    if (i < n) s += in[i];
  }
  __shared__ int sm[32];
  int tot;
  block_exclusive_scan_1024(s, sm, &tot);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void k_scan_single(int* a, int n) {
  __shared__ int sm[32];
  int v[SCAN_ITEMS];
  int s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    int i = threadIdx.x * SCAN_ITEMS + k;
    v[k] = i < n ? a[i] : 0;
    s += v[k];
  }
  int off = block_exclusive_scan_1024(s, sm, nullptr);
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    int i = threadIdx.x * SCAN_ITEMS + k;
    if (i < n) a[i] = off;
    off += v[k];
  }
}

__global__ void k_scan_apply(const int* in, int* out, long n, const int* bsum) {
  __shared__ int sm[32];
  long base = long(blockIdx.x) * SCAN_TILE;
  int v[SCAN_ITEMS];
  int s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    long i = base + long(threadIdx.x) * SCAN_ITEMS + k;
    v[k] = i < n ? in[i] : 0;
    s += v[k];
  }
  __syncthreads();  // in and out may alias: all loads before any store
  int off = block_exclusive_scan_1024(s, sm, nullptr) + bsum[blockIdx.x];
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    long i = base + long(threadIdx.x) * SCAN_ITEMS + k;
    if (i < n) out[i] = off;
    off += v[k];
  }
}

// one tile (n <= SCAN_TILE): the whole scan in one block
__global__ void k_scan_one(const int* in, int* out, int n) {
  __shared__ int sm[32];
  int v[SCAN_ITEMS];
  int s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    int i = threadIdx.x * SCAN_ITEMS + k;
    v[k] = i < n ? in[i] : 0;
    s += v[k];
  }
  __syncthreads();  // in and out may alias: all loads before any store
  int off = block_exclusive_scan_1024(s, sm, nullptr);
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    int i = threadIdx.x * SCAN_ITEMS + k;
    if (i < n) out[i] = off;
    off += v[k];
  }
}

// ---------------------------------------------------------------------------
constexpr int RS_T = 256;       // threads per tile
constexpr int RS_ITEMS = 8;     // items per thread
constexpr int RS_TILE = RS_T * RS_ITEMS;
constexpr int RS_WARPS = RS_T / 32;

// counts of every digit of the passes first .. 7 into total[pass][256]
__global__ void __launch_bounds__(RS_T) k_radix_totals(const uint64_t* __restrict__ keys, long n, int first, int* total) {
  __shared__ int h[8][256];
  for (int i = threadIdx.x; i < 8 * 256; i += RS_T) (&h[0][0])[i] = 0;
  __syncthreads();
  for (long i = long(blockIdx.x) * RS_T + threadIdx.x; i < n; i += long(gridDim.x) * RS_T) {
    const uint64_t k = keys[i];
    for (int p = first; p < 8; ++p) atomicAdd(&h[p][int((k >> (8 * p)) & 0xff)], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 8 * 256; i += RS_T) {
    const int v = (&h[0][0])[i];
    if (v) atomicAdd(total + i, v);
  }
}

// One digit in one launch. A tile publishes its digit counts, then adds up its
// predecessors': from the next one back, eight loads at a time, to the first
// that has published its sum with all before it. Tiles are numbered by a
// ticket, so a tile only waits for blocks that already run and that wait for
// earlier ones alone; the wait is bounded all the same, and a tile that gives
// up counts the keys before it itself. What bounds a pass is the scattered
// write; the histogram and three scan launches of a pass that this replaces
// took as long again (N = 1e5: 15 of 27 us).
//
// A published word: 0 nothing yet, 1 + count for the tile's own count (at most
// RS_TILE), RS_ALL + sum for its sum with all before it (any int fits).
constexpr unsigned RS_ALL = RS_TILE + 2;
static_assert(RS_ALL + 0x7fffffffu > RS_ALL, "a sum of any number of pairs fits a word");
constexpr int RS_LOOK = 8;
constexpr int RS_SPIN = 1 << 20;

__global__ void __launch_bounds__(RS_T)
    k_radix_pass(const uint64_t* kin, const int* vin, uint64_t* kout, int* vout, long n, int shift, const int* total,
                 unsigned* state, int* ticket) {
  __shared__ int wh[RS_WARPS][256];
  __shared__ int base[256];
  __shared__ int s_tile, s_fail, wsum[RS_WARPS];
  if (threadIdx.x == 0) {
    s_tile = atomicAdd(ticket, 1);
    s_fail = 0;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < RS_WARPS * 256; i += RS_T) (&wh[0][0])[i] = 0;
  __syncthreads();
  // warp w owns tile elements [w*256, w*256+256), visited in rounds of 32
  const int tile = s_tile;
  const long wbase = long(tile) * RS_TILE + long(warp) * 32 * RS_ITEMS;
  uint64_t key[RS_ITEMS];
  int val[RS_ITEMS], dig[RS_ITEMS], pos[RS_ITEMS];
  const unsigned lt = (1u << lane) - 1u;
  for (int k = 0; k < RS_ITEMS; ++k) {
    long i = wbase + k * 32 + lane;
    bool ok = i < n;
    key[k] = ok ? kin[i] : 0;
    val[k] = ok ? vin[i] : 0;
    int d = ok ? int((key[k] >> shift) & 0xff) : 256 + lane;  // out-of-range items form singleton groups
    dig[k] = d;
    unsigned peers = __match_any_sync(0xffffffffu, d);
    int rank = __popc(peers & lt);
    int before = ok ? wh[warp][d] : 0;
    __syncwarp();
    pos[k] = before + rank;
    int leader = __ffs(peers) - 1;
    if (ok && lane == leader) wh[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  static_assert(RS_T == 256, "a thread per digit");
  const int d = threadIdx.x;
  // exclusive prefix over warps (warp order = element order), the tile's count
  int cnt = 0;
  for (int w = 0; w < RS_WARPS; ++w) {
    const int c = wh[w][d];
    wh[w][d] = cnt;
    cnt += c;
  }
  volatile unsigned* st = state;
  st[long(tile) * 256 + d] = (tile == 0 ? RS_ALL : 1u) + unsigned(cnt);
  // keys of smaller digits: exclusive sum of the totals
  int x = total[d];
  const int mine = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  int below = x - mine;
  for (int w = 0; w < warp; ++w) below += wsum[w];
  int before = 0;
  if (tile > 0) {
    int t = tile - 1, spins = 0;
    bool found = false;
    while (!found && spins < RS_SPIN) {
      unsigned v[RS_LOOK];
#pragma unroll
      for (int k = 0; k < RS_LOOK; ++k) v[k] = t - k >= 0 ? unsigned(st[long(t - k) * 256 + d]) : unsigned(RS_ALL);
      int used = 0;
#pragma unroll
      for (int k = 0; k < RS_LOOK; ++k)
        if (!found && used == k && v[k] != 0) {
          found = v[k] >= RS_ALL;
          before += int(v[k] - (found ? RS_ALL : 1u));
          ++used;
        }
      t -= used;
      spins = used ? 0 : spins + 1;
    }
    if (!found) s_fail = 1;
  }
  __syncthreads();
  if (s_fail) {
    base[d] = 0;
    __syncthreads();
    for (long i = threadIdx.x; i < long(tile) * RS_TILE; i += RS_T) atomicAdd(&base[int((kin[i] >> shift) & 0xff)], 1);
    __syncthreads();
    before = base[d];
  }
  if (tile > 0) st[long(tile) * 256 + d] = RS_ALL + unsigned(before + cnt);
  base[d] = below + before;
  __syncthreads();
  for (int k = 0; k < RS_ITEMS; ++k) {
    long i = wbase + k * 32 + lane;
    if (i < n) {
      const int dst = base[dig[k]] + wh[warp][dig[k]] + pos[k];
      kout[dst] = key[k];
      vout[dst] = val[k];
    }
  }
}

// Up to SMALL_SORT pairs in one block: a bitonic sort by (key, value), which is
// the stable order when the values come in ascending order or the keys are
// distinct. A thread holds R pairs, block-strided: partners less than 32 apart
// meet by shuffle, up to the block's width through shared memory (one barrier
// a step, two buffers in turn), beyond it in the thread's registers. What
// bounds it is the chain of 55 to 78 steps (all through shared memory it took
// 13 us for 1024 pairs, 54 for 4096; now 8 and 27); the passes above would
// take nine launches.
constexpr int SMALL_SORT = 4096;

template <int R>
__global__ void __launch_bounds__(1024) k_sort_small(uint64_t* keys, int* vals, int n) {
  extern __shared__ uint64_t sm_sort[];  // two buffers of blockDim keys, then of values
  const int T = blockDim.x, t = threadIdx.x;
  uint64_t* sk = sm_sort;
  int* sv = reinterpret_cast<int*>(sm_sort + 2 * T);
  uint64_t key[R];
  int val[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int e = t + i * T;
    key[i] = e < n ? keys[e] : ~uint64_t(0);
    val[i] = e < n ? vals[e] : 0x7fffffff;
  }
  // the smaller or the larger of a pair and its partner
  auto meet = [](uint64_t& k, int& v, uint64_t pk, int pv, bool small) {
    const bool above = k > pk || (k == pk && v > pv);
    if (above == small) k = pk, v = pv;
  };
  int buf = 0;
  for (int k = 2; k <= R * T; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (R > 1 && j >= T) {
        const int x = j / T;
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int h = 0; h < R; ++h)
            if (h == (i ^ x) && i < h) {
              const bool up = ((t + i * T) & k) == 0;
              const uint64_t a = key[i];
              const int av = val[i];
              meet(key[i], val[i], key[h], val[h], up);
              meet(key[h], val[h], a, av, !up);
            }
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int e = t + i * T;
          const bool small = ((e & j) == 0) == ((e & k) == 0);
          uint64_t pk;
          int pv;
          if (j < 32) {
            pk = __shfl_xor_sync(0xffffffffu, key[i], j);
            pv = __shfl_xor_sync(0xffffffffu, val[i], j);
          } else {
            sk[buf * T + t] = key[i];
            sv[buf * T + t] = val[i];
            __syncthreads();
            pk = sk[buf * T + (t ^ j)];
            pv = sv[buf * T + (t ^ j)];
            buf ^= 1;
          }
          meet(key[i], val[i], pk, pv, small);
        }
      }
    }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int e = t + i * T;
    if (e < n) {
      keys[e] = key[i];
      vals[e] = val[i];
    }
  }
}

}  // namespace

size_t scan_scratch_bytes(long n) {
  long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  return size_t(nb + 1) * sizeof(int) + 256;
}

void exclusive_scan(const int* in, int* out, long n, void* scratch, cudaStream_t st) {
  if (n <= 0) return;
  long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nb > SCAN_TILE) throw std::invalid_argument("exclusive_scan: input too long");
  if (nb == 1) {
    k_scan_one<<<1, SCAN_T, 0, st>>>(in, out, int(n));
    PDMK_LAUNCH_CHECK();
    return;
  }
  int* bsum = static_cast<int*>(scratch);
  k_block_sums<<<unsigned(nb), SCAN_T, 0, st>>>(in, n, bsum);
  PDMK_LAUNCH_CHECK();
  k_scan_single<<<1, SCAN_T, 0, st>>>(bsum, int(nb));
  PDMK_LAUNCH_CHECK();
  k_scan_apply<<<unsigned(nb), SCAN_T, 0, st>>>(in, out, n, bsum);
  PDMK_LAUNCH_CHECK();
}

// the totals and tickets of the passes, then every tile's published counts
static size_t radix_state_bytes(long n) {
  const long ntiles = (n + RS_TILE - 1) / RS_TILE;
  return sizeof(int) * (8 * 256 + 64) + size_t(8 * ntiles) * 256 * sizeof(unsigned);
}

size_t radix_sort_scratch_bytes(long n) {
  return size_t(n) * (sizeof(uint64_t) + sizeof(int)) + 768 + radix_state_bytes(n);
}

void radix_sort_pairs(uint64_t* keys, int* vals, long n, int first, void* scratch, cudaStream_t st) {
  if (n <= 1) return;
  if (n <= SMALL_SORT) {
    int pow2 = 32;
    while (pow2 < n) pow2 <<= 1;
    const int T = std::min(1024, pow2);
    auto kern = pow2 <= 1024 ? k_sort_small<1> : pow2 == 2048 ? k_sort_small<2> : k_sort_small<4>;
    kern<<<1, unsigned(T), size_t(2 * T) * (sizeof(uint64_t) + sizeof(int)), st>>>(keys, vals, int(n));
    PDMK_LAUNCH_CHECK();
    return;
  }
  long ntiles = (n + RS_TILE - 1) / RS_TILE;
  char* p = static_cast<char*>(scratch);
  uint64_t* k2 = reinterpret_cast<uint64_t*>(p);
  p += ((size_t(n) * sizeof(uint64_t) + 255) / 256) * 256;
  int* v2 = reinterpret_cast<int*>(p);
  p += ((size_t(n) * sizeof(int) + 255) / 256) * 256;
  int* total = reinterpret_cast<int*>(p);
  int* tickets = total + 8 * 256;
  unsigned* state = reinterpret_cast<unsigned*>(tickets + 64);
  PDMK_CUDA(cudaMemsetAsync(p, 0, radix_state_bytes(n), st));
  k_radix_totals<<<unsigned(std::min<long>(ntiles, 592)), RS_T, 0, st>>>(keys, n, first, total);
  PDMK_LAUNCH_CHECK();
  uint64_t *ka = keys, *kb = k2;
  int *va = vals, *vb = v2;
  for (int pass = first; pass < 8; ++pass) {
    k_radix_pass<<<unsigned(ntiles), RS_T, 0, st>>>(ka, va, kb, vb, n, 8 * pass, total + 256 * pass,
                                                    state + size_t(pass) * ntiles * 256, tickets + pass);
    PDMK_LAUNCH_CHECK();
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (ka != keys) {
    PDMK_CUDA(cudaMemcpyAsync(keys, ka, size_t(n) * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
    PDMK_CUDA(cudaMemcpyAsync(vals, va, size_t(n) * sizeof(int), cudaMemcpyDeviceToDevice, st));
  }
}

}  // namespace pdmk
