// Full-energy kernels (FP64): the plane-wave upward pass, incoming
// expansions, window / difference / residual energies.
//
// Reference counterparts: outgoing_pw_root / outgoing_pw_direct and
// nudft3d1_halfplane (src/planewave.cpp:24-84, include/nudft.hpp:66-123),
// form_incoming_pw (src/planewave.cpp:99-155), eval_energy_window /
// eval_energy_diff / eval_energy_res (src/energy.cpp:21-173).
//
// The outgoing expansion of a box, rho_B(k) = sum_j q_j exp(-i k.x_j) over
// the half grid kz <= 0, is evaluated with box-centred coordinates:
// exp(-i k.x) = exp(-i k.c_B) exp(-i k.(x-c_B)), where k.c_B is an exact
// multiple of pi/3 (k = m dk_l, dk_l bs_l = 2 pi / 3), so the decentring
// factor is an exact sixth root of unity per axis. The charges are real, so
// the centred sums follow from real ones: with f_2m = cos(m dk x) and
// f_2m+1 = sin(m dk x),
//   T[a][b][c] = sum_j q_j f_a(z_j) f_b(y_j) f_c(x_j)
// holds every sign combination of (kz, ky, kx) as sums of eight entries, and
// its (2n+1)^3 entries are half the multiply-adds of the complex products
// over the half grid's (n+1)(2n+1)^2 modes.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "mixed.hpp"
#include "plan.hpp"
#include "tree.hpp"

namespace pdmk {
namespace {

constexpr int TPB = 256;

__device__ inline double block_sum(double v, double* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < nw; ++w) s += sm[w];
  return s;  // valid in thread 0
}

// ---------------------------------------------------------------------------
// T as an FP64 tensor-core product (mma m8n8k4): rows (a, b), columns c,
// summed over particles. Rows come in tiles of eight b for one a, the two a
// (cosine, sine) of one kz together: a warp holds CPW such (kz, b tile) pairs
// against all column tiles, so an A element (one product fz fy) feeds NT
// instructions and a column value 2 CPW. What bounds it: the FP64 pipe, which
// issues tensor instructions at the rate of plain ones (37.1 against 36.6
// TFLOP/s measured on independent chains); per step of four particles a warp
// issues 2 CPW NT of them for 2 CPW products and 3 CPW + NT shared loads.
template <int NK>
struct NudftShape {
  static constexpr int D = 2 * NK + 1;
  static constexpr int N1 = NK + 1;                  // modes per half axis, zero included
  static constexpr int NT = (2 * N1 + 7) / 8;        // tiles of eight entries (four modes) per axis
  static constexpr int PAIRS = N1 * NT;              // (kz, b tile) pairs of a box
  // pairs per warp: accumulators of 8 CPW NT registers, and a last block that
  // is nearly full
  static constexpr int CPW = NT >= 17 ? 1 : NT >= 9 ? 2 : NT >= 7 ? 3 : NT >= 4 ? 5 : NT == 3 ? 7 : NK >= 6 ? 4 : 3;
  static constexpr int WARPS = 4;
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int TILES = (PAIRS + WARPS * CPW - 1) / (WARPS * CPW);  // blocks per item
  // one particle's factors in shared memory: fx, fy, fz; the stride is 4
  // modulo 8, so that the 4 particles x 8 entries of an operand load fall on
  // different banks
  static constexpr int STR = 24 * NT + 4;
  static constexpr int KC = 2 * 32 * STR * 8 <= 100 * 1024 ? 32 : 16;  // particles per chunk
  static constexpr int SMEM = 2 * KC * STR * int(sizeof(double));       // double-buffered
};

// Factors of a chunk's particles into shared memory, one thread per particle
// and axis: cos and sin of m th, m = 0 .. NK, by four interleaved chains of
// steps exp(4 i th) (its own sincos: the chains add roundings, not a drift);
// the charge is folded into fz. Particles past the end get zeros. (A block
// spends about 3 % of its time here; a separate pass wrote and read 1.6 KB
// per particle and level, 2.8 ms at N = 1e6.)
template <int NK>
__device__ __forceinline__ void nudft_factors(const PwItem& w, int base, double* buf, const double* __restrict__ pos,
                                              long stride) {
  using S = NudftShape<NK>;
  for (int t = threadIdx.x; t < S::KC * 3; t += S::THREADS) {
    const int j = t % S::KC, axis = t / S::KC, s = base + j;
    double* dst = buf + j * S::STR + axis * 8 * S::NT;
    if (s >= w.s_end) {
      for (int e = 0; e < 2 * S::N1; ++e) dst[e] = 0.0;
      continue;
    }
    const double x = pos[axis * stride + s] - (axis == 0 ? w.cx : (axis == 1 ? w.cy : w.cz));
    const double sc = axis == 2 ? pos[3 * stride + s] : 1.0;
    const double th = w.dk * x;
    double sn, cs;
    sincos(4.0 * th, &sn, &cs);
    const double2 st = make_double2(cs, sn);
    sincos(th, &sn, &cs);
    const double2 z1 = make_double2(cs, sn);
    double2 v[4];
    v[0] = make_double2(sc, 0.0);
    v[1] = cscale(z1, sc);
    v[2] = cmul(v[1], z1);
    v[3] = cmul(v[2], z1);
#pragma unroll 1
    for (int m = 0; m < S::N1; m += 4)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (m + c < S::N1) {
          *reinterpret_cast<double2*>(dst + 2 * (m + c)) = v[c];
          v[c] = cmul(v[c], st);
        }
  }
}

template <int NK>
__global__ void __launch_bounds__(NudftShape<NK>::THREADS, 2)
    k_nudft(const PwItem* __restrict__ work, const double* __restrict__ pos, long stride) {
  using S = NudftShape<NK>;
  constexpr int NT = S::NT, CPW = S::CPW, STR = S::STR, N1 = S::N1, D = S::D;
  extern __shared__ double smem_d[];
  const PwItem w = work[blockIdx.x / S::TILES];
  const int tile = blockIdx.x % S::TILES;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q4 = lane & 3, q8 = lane >> 2;
  const int g0 = (tile * S::WARPS + warp) * CPW;  // this warp's first pair
  int oz[CPW], oy[CPW];                            // shared-memory offsets of a pair's fz and fy entries
#pragma unroll
  for (int i = 0; i < CPW; ++i) {
    const int g = min(g0 + i, S::PAIRS - 1);
    oz[i] = 16 * NT + 2 * (g / NT);
    oy[i] = 8 * NT + 8 * (g % NT) + q8;
  }
  double acc[CPW][2][NT][2];
#pragma unroll
  for (int i = 0; i < CPW; ++i)
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[i][z][t][0] = acc[i][z][t][1] = 0.0;
  __shared__ double2 roots[6];  // exp(-i pi m / 3)
  if (threadIdx.x < 6) roots[threadIdx.x] = root6(-int(threadIdx.x));
  // the entries past the last mode stay zero
  constexpr int PADN = 8 * NT - 2 * N1;
  if constexpr (PADN > 0)
    for (int t = threadIdx.x; t < 2 * S::KC * 3 * PADN; t += S::THREADS)
      smem_d[(t / (3 * PADN)) * STR + (t / PADN % 3) * 8 * NT + 2 * N1 + t % PADN] = 0.0;
  const int nch = (w.s_end - w.s_begin + S::KC - 1) / S::KC;
  if (nch > 0) nudft_factors<NK>(w, w.s_begin, smem_d, pos, stride);
  __syncthreads();
  for (int ci = 0; ci < nch; ++ci) {
    // the next chunk's factors (its buffer was last read before the barrier
    // that closed the previous iteration)
    if (ci + 1 < nch) nudft_factors<NK>(w, w.s_begin + (ci + 1) * S::KC, smem_d + ((ci + 1) & 1) * S::KC * STR, pos, stride);
    const double* buf = smem_d + (ci & 1) * S::KC * STR + q4 * STR;
    if (g0 < S::PAIRS) {
      // the last chunk of a short box is mostly empty: only its filled steps
      const int steps = min(S::KC / 4, (w.s_end - w.s_begin - ci * S::KC + 3) / 4);
#pragma unroll 1
      for (int ks = 0; ks < steps; ++ks) {
        const double* row = buf + 4 * ks * STR;
        double b[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) b[t] = row[8 * t + q8];
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
          const double y = row[oy[i]];
          const double2 z = *reinterpret_cast<const double2*>(row + oz[i]);
          const double a0 = z.x * y, a1 = z.y * y;
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                : "+d"(acc[i][0][t][0]), "+d"(acc[i][0][t][1])
                : "d"(a0), "d"(b[t]));
            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                : "+d"(acc[i][1][t][0]), "+d"(acc[i][1][t][1])
                : "d"(a1), "d"(b[t]));
          }
        }
      }
    }
    __syncthreads();
  }
  // Epilogue: the four modes (-p, +-q, +-r) of p = |kz|, q = |ky|, r = |kx|. A
  // lane holds the cosine or the sine row of q (lane bit 2), its partner the
  // other; the first takes ky = +q, the second ky = -q.
  const int odd = q8 & 1;
  const double sg = odd ? -1.0 : 1.0;
  const int dx = w.M * (2 * w.X + 1) % 6, dy = w.M * (2 * w.Y + 1) % 6, dz = w.M * (2 * w.Z + 1) % 6;
#pragma unroll
  for (int i = 0; i < CPW; ++i) {
    const int g = g0 + i, p = g / NT, q = 4 * (g % NT) + (q8 >> 1);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      double own[4], oth[4];  // [kz cosine, sine][kx cosine, sine]
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        own[v] = acc[i][v >> 1][t][v & 1];
        oth[v] = __shfl_xor_sync(0xffffffffu, own[v], 4);
      }
      const int r = 4 * t + q4;
      if (g < S::PAIRS && q < N1 && r < N1 && !(odd && q == 0)) {
        // y cosine and y sine entries
        double c[4], sv[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          c[v] = odd ? oth[v] : own[v];
          sv[v] = odd ? own[v] : oth[v];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h == 1 && r == 0) continue;
          const double ta = h ? -1.0 : 1.0;  // kx = ta r
          const double st = sg * ta;
          const double a1 = c[0] - st * sv[1], b1 = sg * sv[0] + ta * c[1];
          const double a2 = c[2] - st * sv[3], b2 = sg * sv[2] + ta * c[3];
          const int ky = odd ? -q : q, kx = h ? -r : r;
          const double2 v = cmul(make_double2(a1 + b2, a2 - b1), roots[unsigned(dx * kx + dy * ky - dz * p + 30 * NK) % 6u]);
          w.out[(size_t(NK - p) * D + NK + ky) * D + NK + kx] = v;
        }
      }
    }
  }
}

template <int NK>
void launch_nudft(const PwItem* d_work, int nwork, const double* pos, long stride, cudaStream_t st) {
  using S = NudftShape<NK>;
  if (nwork == 0) return;
  // per device and thread-safe: replica energies call this from several host threads
  raise_smem_limit(reinterpret_cast<const void*>(k_nudft<NK>), S::SMEM);
  k_nudft<NK><<<unsigned(nwork) * S::TILES, S::THREADS, S::SMEM, st>>>(d_work, pos, stride);
  PDMK_LAUNCH_CHECK();
}

// blocks of an item
int nudft_tiles(int nk) {
  switch (nk) {
    case 4: return NudftShape<4>::TILES;
    case 6: return NudftShape<6>::TILES;
    case 8: return NudftShape<8>::TILES;
    case 12: return NudftShape<12>::TILES;
    case 13: return NudftShape<13>::TILES;
    case 17: return NudftShape<17>::TILES;
    case 19: return NudftShape<19>::TILES;
    case 26: return NudftShape<26>::TILES;
    case 32: return NudftShape<32>::TILES;  // Ewald structure factor, level 2
    case 64: return NudftShape<64>::TILES;  // Ewald structure factor, level 3
    default: throw std::invalid_argument("unsupported mode count");
  }
}

void dispatch_nudft(int nk, const PwItem* d_work, int nwork, const double* pos, long stride, cudaStream_t st) {
  switch (nk) {
    case 4: launch_nudft<4>(d_work, nwork, pos, stride, st); break;
    case 6: launch_nudft<6>(d_work, nwork, pos, stride, st); break;
    case 8: launch_nudft<8>(d_work, nwork, pos, stride, st); break;
    case 12: launch_nudft<12>(d_work, nwork, pos, stride, st); break;
    case 13: launch_nudft<13>(d_work, nwork, pos, stride, st); break;
    case 17: launch_nudft<17>(d_work, nwork, pos, stride, st); break;
    case 19: launch_nudft<19>(d_work, nwork, pos, stride, st); break;
    case 26: launch_nudft<26>(d_work, nwork, pos, stride, st); break;
    case 32: launch_nudft<32>(d_work, nwork, pos, stride, st); break;
    case 64: launch_nudft<64>(d_work, nwork, pos, stride, st); break;
    default: throw std::invalid_argument("unsupported mode count");
  }
}

// sum split-K chunk partials of box b into its output: 256 / ROWS modes x ROWS
// chunk lanes a block, four loads in flight a thread. Eight lanes where there are
// many chunks (the 592 of a small root: 11 us, a lane per mode 47), one where
// there are few (64 boxes of two chunks, N = 1e6: 15 us, eight lanes 57).
template <int ROWS>
__global__ void __launch_bounds__(256) k_reduce_chunks(const double2* __restrict__ part,
                                                       const PwSplit* __restrict__ split, int H) {
  constexpr int MODES = 256 / ROWS;
  __shared__ double2 sm[ROWS][MODES];
  const PwSplit b = split[blockIdx.y];
  const int lane = threadIdx.x % MODES, row = threadIdx.x / MODES;
  const int k = blockIdx.x * MODES + lane;
  const double2* p = part + size_t(b.first) * H + k;
  double2 s[4] = {};
  if (k < H)
    for (int c = row; c < b.n; c += 4 * ROWS) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + ROWS * u < b.n) s[u] = cadd(s[u], p[size_t(c + ROWS * u) * H]);
    }
  double2 t = cadd(cadd(s[0], s[1]), cadd(s[2], s[3]));
  if (ROWS > 1) {
    sm[row][lane] = t;
    __syncthreads();
    if (row > 0) return;
#pragma unroll
    for (int r = 1; r < ROWS; ++r) t = cadd(t, sm[r][lane]);
  }
  if (k < H) b.out[k] = t;
}

// n_split boxes with n_items partials in all
void launch_reduce_chunks(const double2* part, const PwSplit* split, int n_split, long n_items, int H, cudaStream_t st) {
  if (n_split == 0) return;
  const bool many = n_items >= 16L * n_split;
  auto kern = many ? k_reduce_chunks<8> : k_reduce_chunks<1>;
  const int modes = many ? 32 : 256;
  kern<<<dim3(unsigned((H + modes - 1) / modes), unsigned(n_split)), 256, 0, st>>>(part, split, H);
  PDMK_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// inc_B = conj(out_B) + sum_C conj(out_C * exp(-i k.p L)) over B's 26
// colleagues C (form_incoming_pw, src/planewave.cpp:99-155), for the
// 4 x 4 x 4 boxes of level l below one box G of level l - 2 at once: their
// 27-box neighbourhoods lie in the 6 x 6 x 6 cube of level-l cells around
// them. Per tile of INC_KT modes a block sums in two steps: a thread loads the
// six z cells of a column, all at once, and leaves its four 3-cell z sums in
// shared memory; then a thread adds 3 y neighbours of them for the six x and
// slides the 3-wide x window over the result for 4 receivers. (Staging the raw
// cells and summing 3 x 3 neighbourhoods from them moved twice the
// shared-memory words, and the loads waited behind them.) Cells next to no
// receiver are not loaded and columns without a needed cell are left out: in
// the deep levels of a clustered tree a cube holds one or two receivers. The
// periodic image phases are cube roots of unity, separable over the axes, so
// they are applied to the sums at the cube's faces. The energy partial of a
// block sums its non-leaf receivers, which share one level.
constexpr int INC_KT = 16;    // modes per tile
constexpr int INC_T = 288;    // threads: INC_KT modes x 18 columns, half of a full cube's
constexpr int INC_CELLS = 216;
constexpr size_t INC_SMEM = sizeof(double2) * INC_KT * (4 * 36 + 64);  // z sums, the receivers' own rows

// rank of a refined cell within its level (Morton order)
__device__ inline int refined_rank(const DevTree& T, int level, uint64_t cell) {
  const uint32_t w = T.bm_d[level][cell >> 5];
  return T.wprefix_d[level][cell >> 5] + __popc(w & ((1u << (cell & 31)) - 1u));
}

// v exp(-2 pi i e / 3)
__device__ __forceinline__ double2 rot3(double2 v, int e) {
  if (e == 0) return v;
  const double h = e == 1 ? -0.86602540378443864676 : 0.86602540378443864676;
  return make_double2(-0.5 * v.x - h * v.y, -0.5 * v.y + h * v.x);
}

// Block (slot, c) of slots x ncubes handles the tiles slot, slot + slots, ... of
// cube c, so its set-up (the cube's cell lookup) is paid once, and the cubes
// sharing a slot walk the same tiles together (the cells two neighbouring cubes
// share meet in L2). part: the blocks' energy partials, or null; touched: only
// cubes with a marked cell, or null.
template <int NK>
__device__ __forceinline__ void incoming_cube(const DevTree& T, const int* __restrict__ cubes, int ncubes, int slots,
                                              double* part, const int* __restrict__ touched) {
  constexpr int D = 2 * NK + 1, H = (NK + 1) * D * D;
  extern __shared__ double2 zs[];            // z sums [z][cy][cx][INC_KT]
  double2* own = zs + 4 * 36 * INC_KT;       // the receivers' own rows [receiver][INC_KT]
  __shared__ int s_row[INC_CELLS];           // outgoing row of each cell, -1: absent, empty or not needed
  __shared__ int s_recv[64];                 // expansion row of each receiver, -1: none
  __shared__ int s_col[36], s_line[16];      // columns (cx + 6 cy) and receiver lines (y + 4 z) with something to do
  __shared__ int s_ncol, s_nline, s_any;
  __shared__ double sm[32];
  const int slot = blockIdx.x / ncubes, cb = blockIdx.x % ncubes;
  const int G = cubes[cb];
  const int l = T.node_level[G] + 2;
  const int side = 1 << l;
  const uint64_t gp = T.node_prefix[G];
  const int O[3] = {4 * int(compact3(gp)), 4 * int(compact3(gp >> 1)), 4 * int(compact3(gp >> 2))};
  const int base = T.pw_base;
  const int tid = threadIdx.x;
  if (tid == 0) s_any = 0;
  __syncthreads();
  if (tid < INC_CELLS) {
    const int c[3] = {tid % 6 - 1, (tid / 6) % 6 - 1, tid / 36 - 1};
    int g[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int v = O[a] + c[a];
      g[a] = v < 0 ? v + side : (v >= side ? v - side : v);
    }
    const uint64_t m = morton3(uint32_t(g[0]), uint32_t(g[1]), uint32_t(g[2]));
    int node = -1;
    if ((T.bm_d[l - 1][m >> 8] >> ((m >> 3) & 31)) & 1u)
      node = T.level_start_d[l] + 8 * refined_rank(T, l - 1, m >> 3) + int(m & 7);
    s_row[tid] = (node >= 0 && T.node_count[node] > 0) ? node - base : -1;
    if (c[0] >= 0 && c[0] < 4 && c[1] >= 0 && c[1] < 4 && c[2] >= 0 && c[2] < 4)
      s_recv[c[0] + 4 * c[1] + 16 * c[2]] = (node >= 0 && T.node_child0[node] >= 0) ? node - base : -1;
    if (touched && node >= 0 && touched[node - base] != 0) s_any = 1;
  }
  __syncthreads();
  // after a sequence of moves: nothing to do when no outgoing row of the cube changed
  if (touched && !s_any) return;
  if (touched && tid < 32 && slot == 0) {
    int n = (s_recv[tid] >= 0) + (s_recv[tid + 32] >= 0);
    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
    if (tid == 0) atomicAdd(&T.work[1], 32ull * H * (unsigned long long)n);
  }
  // which cells lie next to a receiver, the columns that hold one, and the
  // lines with a receiver
  {
    bool need = false;
    if (tid < INC_CELLS) {
      const int c[3] = {tid % 6 - 1, (tid / 6) % 6 - 1, tid / 36 - 1};
      for (int z = max(c[2] - 1, 0); z <= min(c[2] + 1, 3); ++z)
        for (int y = max(c[1] - 1, 0); y <= min(c[1] + 1, 3); ++y)
          for (int x = max(c[0] - 1, 0); x <= min(c[0] + 1, 3); ++x) need = need || s_recv[x + 4 * y + 16 * z] >= 0;
    }
    __syncthreads();
    if (tid < INC_CELLS && !need) s_row[tid] = -2;
    __syncthreads();
    if (tid < 32) {
      int n = 0;
      for (int b = 0; b < 36; b += 32) {
        bool on = false;
        if (b + tid < 36)
          for (int z = 0; z < 6; ++z) on = on || s_row[z * 36 + b + tid] != -2;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) s_col[n + __popc(m & ((1u << tid) - 1u))] = b + tid;
        n += __popc(m);
      }
      bool on = false;
      if (tid < 16)
        for (int x = 0; x < 4; ++x) on = on || s_recv[x + 4 * tid] >= 0;
      const unsigned m = __ballot_sync(0xffffffffu, on);
      if (on) s_line[__popc(m & ((1u << tid) - 1u))] = tid;
      if (tid == 0) {
        s_ncol = n;
        s_nline = __popc(m);
      }
    }
    __syncthreads();
  }
  const int ncol = s_ncol, nline = s_nline;
  const int two_l = (l & 1) ? 2 : 1;
  // the cube's faces that lie on the box's: the cells there are images
  bool lo_face[3], hi_face[3];
  for (int a = 0; a < 3; ++a) {
    lo_face[a] = O[a] == 0;
    hi_face[a] = O[a] + 4 == side;
  }
  const int kk = tid % INC_KT;
  double e = 0;
  constexpr int ktiles = (H + INC_KT - 1) / INC_KT;
  for (int tile = slot; tile < ktiles; tile += slots) {
    const int k = tile * INC_KT + kk;
    const bool kin = k < H;
    // the image phase is exp(-2 pi i e / 3) with e = sum over axes of
    // f (i - n) 2^l mod 3 (f = -1 below, +1 above)
    const int ix = k % D, iy = (k / D) % D, iz = k / (D * D);
    const int ex = (((ix - NK) % 3 + 3) * two_l) % 3, ey = (((iy - NK) % 3 + 3) * two_l) % 3,
              ez = (((iz - NK) % 3 + 3) * two_l) % 3;
    // two columns a thread, the loads of both before the first is used
    for (int c0 = tid / INC_KT; c0 < ncol; c0 += 2 * (INC_T / INC_KT)) {
      double2 v[2][6];
      int col[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int ci = c0 + j * (INC_T / INC_KT);
        col[j] = ci < ncol ? s_col[ci] : -1;
#pragma unroll
        for (int z = 0; z < 6; ++z) {
          const int row = col[j] >= 0 ? s_row[z * 36 + col[j]] : -1;
          v[j][z] = (row >= 0 && kin) ? T.out[size_t(row) * H + k] : make_double2(0.0, 0.0);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (col[j] < 0) break;
        const int cx = col[j] % 6, cy = col[j] / 6;
        if (cx >= 1 && cx <= 4 && cy >= 1 && cy <= 4)
#pragma unroll
          for (int z = 0; z < 4; ++z) own[(cx - 1 + 4 * (cy - 1) + 16 * z) * INC_KT + kk] = v[j][z + 1];
        if (lo_face[2]) v[j][0] = rot3(v[j][0], (3 - ez) % 3);
        if (hi_face[2]) v[j][5] = rot3(v[j][5], ez);
#pragma unroll
        for (int z = 0; z < 4; ++z) zs[(z * 36 + col[j]) * INC_KT + kk] = cadd(cadd(v[j][z], v[j][z + 1]), v[j][z + 2]);
      }
    }
    __syncthreads();
    for (int li = tid / INC_KT; li < nline; li += INC_T / INC_KT) {
      const int line = s_line[li], ry = line & 3, rz = line >> 2;
      double2 c[6];
#pragma unroll
      for (int cx = 0; cx < 6; ++cx) {
        const double2* p = zs + (rz * 36 + ry * 6 + cx) * INC_KT + kk;
        double2 a = p[0], b = p[12 * INC_KT];
        if (ry == 0 && lo_face[1]) a = rot3(a, (3 - ey) % 3);
        if (ry == 3 && hi_face[1]) b = rot3(b, ey);
        c[cx] = cadd(cadd(a, p[6 * INC_KT]), b);
      }
      if (lo_face[0]) c[0] = rot3(c[0], (3 - ex) % 3);
      if (hi_face[0]) c[5] = rot3(c[5], ex);
      if (kin) {
        const double d2 = T.D2[k];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int rrow = s_recv[x + 4 * line];
          if (rrow < 0) continue;
          const double2 inc = cconj(cadd(cadd(c[x], c[x + 1]), c[x + 2]));
          T.inc[size_t(rrow) * H + k] = inc;
          const double2 o = own[(x + 4 * line) * INC_KT + kk];
          e += (o.x * inc.x - o.y * inc.y) * d2;
        }
      }
    }
    __syncthreads();
  }
  if (!part) return;
  double s = block_sum(e, sm);
  if (tid == 0) part[blockIdx.x] = s;
}

template <int NK>
__global__ void __launch_bounds__(INC_T, 3) k_incoming_cube(DevTree T, const int* __restrict__ cubes, int ncubes,
                                                             int slots, double* part,
                                                             const int* __restrict__ touched) {
  incoming_cube<NK>(T, cubes, ncubes, slots, part, touched);
}

// the touched cubes of a set of trees
template <int NK>
__global__ void __launch_bounds__(INC_T, 3) k_incoming_cubes(const DevTree* __restrict__ trees,
                                                              const SequenceRows* __restrict__ rows, int n) {
  const int t = set_tree();
  if (t >= n) return;
  const SequenceRows r = rows[t];
  if (int(blockIdx.x) >= r.slots * r.n_cubes || *r.n_list == 0) return;
  incoming_cube<NK>(trees[t], r.cubes, r.n_cubes, r.slots, nullptr, r.touched);
}

template <int NK>
void launch_incoming_nk(const DevTree& D, const int* cubes, int ncubes, int slots, double* part, const int* touched,
                        cudaStream_t st) {
  raise_smem_limit(reinterpret_cast<const void*>(k_incoming_cube<NK>), INC_SMEM);
  k_incoming_cube<NK><<<unsigned(slots * ncubes), INC_T, INC_SMEM, st>>>(D, cubes, ncubes, slots, part, touched);
  PDMK_LAUNCH_CHECK();
}

void launch_incoming(const DevTree& D, const int* cubes, int ncubes, int slots, double* part, const int* touched,
                     cudaStream_t st) {
  switch (D.n_diff) {
    case 4: launch_incoming_nk<4>(D, cubes, ncubes, slots, part, touched, st); break;
    case 6: launch_incoming_nk<6>(D, cubes, ncubes, slots, part, touched, st); break;
    case 8: launch_incoming_nk<8>(D, cubes, ncubes, slots, part, touched, st); break;
    case 12: launch_incoming_nk<12>(D, cubes, ncubes, slots, part, touched, st); break;
    case 13: launch_incoming_nk<13>(D, cubes, ncubes, slots, part, touched, st); break;
    case 17: launch_incoming_nk<17>(D, cubes, ncubes, slots, part, touched, st); break;
    case 19: launch_incoming_nk<19>(D, cubes, ncubes, slots, part, touched, st); break;
    case 26: launch_incoming_nk<26>(D, cubes, ncubes, slots, part, touched, st); break;
    default: throw std::invalid_argument("incoming pass: unsupported mode count");
  }
}

template <int NK>
void launch_incoming_set_nk(const DevTree* trees, const SequenceRows* rows, int n_trees, int blocks, cudaStream_t st) {
  raise_smem_limit(reinterpret_cast<const void*>(k_incoming_cubes<NK>), INC_SMEM);
  k_incoming_cubes<NK><<<set_grid(blocks, n_trees), INC_T, INC_SMEM, st>>>(trees, rows, n_trees);
  PDMK_LAUNCH_CHECK();
}

// E_diff from the cube-tiled partials: sum over cubes C_l dscale_l
// sum_slots part, minus sum over non-leaf boxes Q_B S_l
__global__ void k_diff_finish_cube(DevTree T, const int* __restrict__ cubes, int ncubes, int slots,
                                   const double* part, const int* __restrict__ boxes, int nboxes, const double* q2,
                                   const double* Cl, const double* Sl, double* out) {
  __shared__ double sm[32];
  double e = 0;
  // all (slot, cube) terms over the threads: a small tree has one cube of 500
  // slots, which one thread summed in 28 us
  for (int i = threadIdx.x; i < slots * ncubes; i += blockDim.x) {
    const int l = T.node_level[cubes[i % ncubes]] + 2;
    e += Cl[l] * level_dscale(l) * part[i];
  }
  for (int b = threadIdx.x; b < nboxes; b += blockDim.x) e -= q2[b] * Sl[T.node_level[boxes[b]]];
  double s = block_sum(e, sm);
  if (threadIdx.x == 0) {
    *out = s;
    T.counter[15] = 1;  // the incoming rows are written
  }
}

// Re sum out_B inc_B D_2 per (box, k tile) on the stored incoming expansions
__global__ void k_tridot(DevTree T, const int* __restrict__ boxes, int nboxes, double* part) {
  __shared__ double sm[32];
  const int tile = blockIdx.x / nboxes, b = blockIdx.x % nboxes;
  const int node = boxes[b];
  const int k = tile * blockDim.x + threadIdx.x;
  const int base = T.pw_base;
  double e = 0;
  if (k < T.H) {
    double2 o = T.out[size_t(node - base) * T.H + k];
    double2 c = T.inc[size_t(node - base) * T.H + k];
    e = (o.x * c.x - o.y * c.y) * T.D2[k];
  }
  double s = block_sum(e, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// sum of q^2 over each box's slots
__global__ void k_box_q2(DevTree T, const int* __restrict__ boxes, double* q2) {
  __shared__ double sm[32];
  int node = boxes[blockIdx.x];
  double v = 0;
  for (int s = T.node_begin[node] + threadIdx.x; s < T.node_end[node]; s += blockDim.x) v += T.sq[s] * T.sq[s];
  double tot = block_sum(v, sm);
  if (threadIdx.x == 0) q2[blockIdx.x] = tot;
}

// E_diff = sum_box [C_l dscale_l sum_tiles part - Q_B S_l]
__global__ void k_diff_finish(DevTree T, const int* __restrict__ boxes, int nboxes, int ktiles, const double* part,
                              const double* q2, const double* Cl, const double* Sl, double* out) {
  __shared__ double sm[32];
  double e = 0;
  for (int b = threadIdx.x; b < nboxes; b += blockDim.x) {
    int node = boxes[b];
    int l = T.node_level[node];
    double t = 0;
    for (int tile = 0; tile < ktiles; ++tile) t += part[size_t(tile) * nboxes + b];
    e += Cl[l] * level_dscale(l) * t - q2[b] * Sl[l];
  }
  double s = block_sum(e, sm);
  if (threadIdx.x == 0) *out = s;
}

// window energy; the self term sum(q^2) psi_0(0) / (2 b_2 C0) takes sum(q^2)
// from the device (q2) so that no host round trip is needed
__global__ void k_window(DevTree T, double scale, const double* q2, double psi0_0, double self_den, double* out) {
  __shared__ double sm[32];
  double e = 0;
  for (int k = threadIdx.x; k < T.Hw; k += blockDim.x) {
    double2 o = T.out_root[k];
    e += (o.x * o.x + o.y * o.y) * T.W[k];
  }
  double s = block_sum(e, sm);
  if (threadIdx.x == 0) *out = s * scale - *q2 * psi0_0 / self_den;
}


__device__ inline int periodic_shift_d(double xi, double xj, double L, double bi, double bj) {
  if (xi < bi && xj > (L - bj)) return 1;
  if (xi > (L - bi) && xj < bj) return -1;
  return 0;
}

__device__ inline void node_center(const DevTree& T, int node, double* c) {
  uint64_t p = T.node_prefix[node];
  int l = T.node_level[node];
  double scale = ldexp(1.0, -l);
  c[0] = T.L * (double(compact3(p)) * scale + 0.5 * scale);
  c[1] = T.L * (double(compact3(p >> 1)) * scale + 0.5 * scale);
  c[2] = T.L * (double(compact3(p >> 2)) * scale + 0.5 * scale);
}

constexpr int RES_T = 128;
constexpr int RES_TCH = 64;   // targets of one work item
constexpr int RES_SCH = 256;  // sources staged in shared memory per round

// the smallest and largest of a full warp's values (one instruction on sm_100)
__device__ __forceinline__ float warp_min(float a) {
  float d;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(a));
  return d;
}
__device__ __forceinline__ float warp_max(float a) {
  float d;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(a));
  return d;
}
// two FP32 values in one 64-bit register (sm_100's packed arithmetic)
__device__ __forceinline__ unsigned long long both_f32x2(float a) {
  const unsigned long long w = __float_as_uint(a);
  return w << 32 | w;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// leaf near field: 1/2 sum_{i in B} q_i sum_{j in N(B), j != i} q_j res(r_ij; bs_B)
// (eval_energy_res, src/energy.cpp:82-173). One block per (leaf, chunk of
// RES_TCH targets), so a large leaf is spread over several blocks; leaves are
// listed coarse level first, so the big items start first. The up to 35
// source boxes (self, colleagues, coarse-grain) are flattened into one index
// range, staged in rounds of RES_SCH with their periodic offsets applied.
//
// About one pair in six lies inside the cut-off. Testing all of them in FP64
// took most of the kernel's instructions, so the pairs are sieved first: a
// warp holds 32 targets, which are neighbours in Morton order (as a tile of 32
// sources is), and skips the tiles whose bounding box is out of reach; the
// pairs left are tested in FP32 with a margin above its rounding, and the ones
// that may be inside go to the warp's queue as (target, source) indices, a
// tile's at once: a lane keeps its target's 32 answers as a bit mask (nine
// instructions a pair, where asking the warp for every pair took 28). The
// queue is evaluated 32 pairs at a time in FP64, distance and polynomial, so
// the sum is the one over all pairs (a pair beyond the cut-off adds zero there).
//
// MINB, resident blocks: filled tiles want registers (N = 1e5, 55 particles a
// leaf: 0.46 ms at 7 blocks, 0.49 at 8, 0.54 at 9), small leaves want blocks to
// hide the staging behind (N = 1e6, 30 a leaf: 1.04 ms at 7, 1.00 at 8, 0.92 at
// 9).
template <int NP, int MINB>
__global__ void __launch_bounds__(RES_T, MINB) k_residual(DevTree T, const int* __restrict__ leaves, int ny,
                                                    double* part) {
  __shared__ double ux[RES_SCH], uy[RES_SCH], uz[RES_SCH], uq[RES_SCH];
  // negated coordinates relative to the leaf's centre, in box sides
  __shared__ __align__(16) float ufx[RES_SCH], ufy[RES_SCH], ufz[RES_SCH];
  __shared__ float t_lo[RES_SCH / 32][3], t_hi[RES_SCH / 32][3];  // bounding boxes of the source tiles
  __shared__ double gx[RES_TCH], gy[RES_TCH], gz[RES_TCH], gq[RES_TCH];
  __shared__ int m_beg[36], m_pre[37];
  __shared__ double m_off[36][3], m_w[36];
  __shared__ double sm[32];
  __shared__ unsigned short q_pair[RES_T / 32][1056];  // per warp: at most 31 pairs waiting and a tile's 1024
  const ResidualPoly<NP> poly(T);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int node = leaves[blockIdx.x / ny], chunk = blockIdx.x % ny;
  const int l = T.node_level[node];
  const int cnt = T.leaf_count[node];
  double e = 0;
  if (l >= 2 && cnt > chunk * RES_TCH) {
    const double b = level_box(T, l), inv_b = 1.0 / b;
    // FP32 coordinates in units of b (any box size is in their range) reach 2.5
    // from the centre: each is off by 2^-23 at most, a squared distance near 1 by
    // less than 2e-6
    const float cut = 1.0f + 8e-6f;
    const float far = 1e18f;  // where a lane without a target, or a tile's empty place, is put
    const int tb = T.node_begin[node];
    double ci[3];
    node_center(T, node, ci);
    if (threadIdx.x < 36) {
      const int src = threadIdx.x;
      int j = -1;
      if (src == 0) j = node;
      else if (src <= 27) j = (src - 1 == 13) ? -1 : T.col27[size_t(node) * 27 + (src - 1)];
      else j = T.coarse8[size_t(node) * 8 + (src - 28)];
      // A pair of particles in two leaves of the same level meets the same
      // cut-off from either side, so only the leaf with the smaller id sums
      // it, with weight 2. Other sources (non-leaf colleagues, coarser
      // neighbours) see a cut-off that depends on the target's level: both
      // sides sum those.
      const bool same_level_leaf = src >= 1 && src <= 27 && j >= 0 && T.node_child0[j] < 0;
      const bool skip = same_level_leaf && j < node;
      int beg = 0, n = 0;
      double off[3] = {0, 0, 0};
      if (j >= 0 && !skip && T.node_count[j] > 0) {
        double cj[3];
        node_center(T, j, cj);
        const double bj = level_box(T, T.node_level[j]);
        for (int dd = 0; dd < 3; ++dd) off[dd] = -periodic_shift_d(ci[dd], cj[dd], T.L, b, bj) * T.L;
        beg = T.node_begin[j];
        n = (T.node_child0[j] < 0 ? beg + T.leaf_count[j] : T.node_end[j]) - beg;
      }
      m_beg[src] = beg;
      m_pre[src] = n;
      m_w[src] = same_level_leaf ? 2.0 : 1.0;
      for (int dd = 0; dd < 3; ++dd) m_off[src][dd] = off[dd];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = 0;
      for (int src = 0; src < 36; ++src) {
        const int n = m_pre[src];
        m_pre[src] = s;
        s += n;
      }
      m_pre[36] = s;
    }
    __syncthreads();
    const int total = m_pre[36];
    for (int t0 = chunk * RES_TCH; t0 < cnt; t0 += ny * RES_TCH) {
      const int nt = min(RES_TCH, cnt - t0);
      // groups of 32 targets, the warps of one group sharing the source tiles
      const int ngrp = nt <= 32 ? 1 : 2, nparts = RES_T / 32 / ngrp;
      const int grp = wid % ngrp, sp = wid / ngrp;
      const int it = grp * 32 + lane;
      if (threadIdx.x < nt) {
        const int s = tb + t0 + threadIdx.x;
        gx[threadIdx.x] = T.sx[s];
        gy[threadIdx.x] = T.sy[s];
        gz[threadIdx.x] = T.sz[s];
        gq[threadIdx.x] = T.sq[s];
      }
      __syncthreads();
      const bool act = it < nt;
      const float fx = act ? float((gx[it] - ci[0]) * inv_b) : far, fy = act ? float((gy[it] - ci[1]) * inv_b) : far,
                  fz = act ? float((gz[it] - ci[2]) * inv_b) : far;
      const unsigned long long fx2 = both_f32x2(fx), fy2 = both_f32x2(fy), fz2 = both_f32x2(fz);
      const unsigned long long ncut2 = both_f32x2(-cut);
      float lo[3] = {fx, fy, fz}, hi[3] = {act ? fx : -far, act ? fy : -far, act ? fz : -far};
#pragma unroll
      for (int a = 0; a < 3; ++a) lo[a] = warp_min(lo[a]), hi[a] = warp_max(hi[a]);
      for (int u0 = 0; u0 < total; u0 += RES_SCH) {
        const int ns = min(RES_SCH, total - u0);
        __syncthreads();
        for (int t = threadIdx.x; t < (ns + 31) / 32 * 32; t += blockDim.x) {  // whole warps
          float f[3] = {-far, -far, -far};  // far from everything, from an absent target too
          float flo[3] = {far, far, far}, fhi[3] = {-far, -far, -far};
          if (t < ns) {
            const int ei = u0 + t;
            int a = 0, z = 36;  // largest src with m_pre[src] <= ei
            while (z - a > 1) {
              const int mid = (a + z) >> 1;
              if (m_pre[mid] <= ei) a = mid;
              else z = mid;
            }
            const int s = m_beg[a] + (ei - m_pre[a]);
            const double x = T.sx[s] + m_off[a][0], y = T.sy[s] + m_off[a][1], zz = T.sz[s] + m_off[a][2];
            ux[t] = x;
            uy[t] = y;
            uz[t] = zz;
            uq[t] = T.sq[s] * m_w[a];
            f[0] = float((x - ci[0]) * inv_b), f[1] = float((y - ci[1]) * inv_b), f[2] = float((zz - ci[2]) * inv_b);
#pragma unroll
            for (int a2 = 0; a2 < 3; ++a2) flo[a2] = fhi[a2] = f[a2];
          }
          ufx[t] = -f[0];
          ufy[t] = -f[1];
          ufz[t] = -f[2];
#pragma unroll
          for (int a = 0; a < 3; ++a) flo[a] = warp_min(flo[a]), fhi[a] = warp_max(fhi[a]);
          if (lane < 3) {
            t_lo[t >> 5][lane] = lane == 0 ? flo[0] : lane == 1 ? flo[1] : flo[2];
            t_hi[t >> 5][lane] = lane == 0 ? fhi[0] : lane == 1 ? fhi[1] : fhi[2];
          }
        }
        __syncthreads();
        int qn = 0;  // pairs waiting in this warp's queue (warp-uniform)
        auto evaluate = [&](int at, int n) {  // n queued pairs from place `at`
          if (lane < n) {
            const int p = q_pair[wid][at + lane];
            const int js = p & 255, i = p >> 8;
            const double dx = gx[i] - ux[js], dy = gy[i] - uy[js], dz = gz[i] - uz[js];
            const double r2 = dx * dx + dy * dy + dz * dz;
            e += gq[i] * uq[js] * poly.from_r2(r2, inv_b);  // zero at r = 0 (the target itself) and beyond the cut-off
          }
        };
        for (int tile = sp; tile * 32 < ns; tile += nparts) {
          float d2 = 0.0f;
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const float d = fmaxf(0.0f, fmaxf(lo[a] - t_hi[tile][a], t_lo[tile][a] - hi[a]));
            d2 = fmaf(d, d, d2);
          }
          if (d2 > cut) continue;
          // r^2 - cut for two sources at a time (packed FP32), its sign the
          // answer: source j ends up at bit 31 - j
          unsigned mask = 0;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const ulonglong2 sx = *reinterpret_cast<const ulonglong2*>(ufx + tile * 32 + j);
            const ulonglong2 sy = *reinterpret_cast<const ulonglong2*>(ufy + tile * 32 + j);
            const ulonglong2 sz = *reinterpret_cast<const ulonglong2*>(ufz + tile * 32 + j);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const unsigned long long dx = add_f32x2(fx2, h ? sx.y : sx.x), dy = add_f32x2(fy2, h ? sy.y : sy.x),
                                       dz = add_f32x2(fz2, h ? sz.y : sz.x);
              const unsigned long long r = fma_f32x2(dz, dz, fma_f32x2(dy, dy, fma_f32x2(dx, dx, ncut2)));
              mask = __funnelshift_l(unsigned(r), mask, 1);
              mask = __funnelshift_l(unsigned(r >> 32), mask, 1);
            }
          }
          // this lane's places in the queue: after the pairs waiting and the lanes below
          const int mine = __popc(mask);
          int at = mine;
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += y;
          }
          const int all = __shfl_sync(0xffffffffu, at, 31);
          at += qn - mine;
          while (mask) {
            const int j = __clz(mask);
            q_pair[wid][at++] = static_cast<unsigned short>((it << 8) | (tile * 32 + j));
            mask &= ~(0x80000000u >> j);
          }
          qn += all;
          __syncwarp();
          int done = 0;
          for (; qn - done >= 32; done += 32) evaluate(done, 32);
          qn -= done;
          unsigned short left = 0;  // the rest moves to the front
          if (lane < qn) left = q_pair[wid][done + lane];
          __syncwarp();
          if (lane < qn) q_pair[wid][lane] = left;
        }
        __syncwarp();
        evaluate(0, qn);  // the queue names places of this round's sources
      }
      __syncthreads();  // the targets are replaced
    }
  }
  double s = block_sum(0.5 * e, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// ---------------------------------------------------------------------------
// FP64 Ewald comparator (the reference's Ewald summation, src/ewald.cpp:17-223):
// E = 1/2 sum_{i != j, images} q_i q_j erfc(alpha r)/r
//   + (2 pi / V) sum_{k != 0} exp(-k^2 / (4 alpha^2)) / k^2 |S(k)|^2
//   - alpha / sqrt(pi) sum_i q_i^2,  S(k) = sum_j q_j exp(i k.r_j).
// The real-space cut-off is the box size of one tree level, so the 27 boxes
// of that level around a box hold every pair; S(k) comes from the NUDFT
// kernel (the conjugate, which leaves |S|^2 unchanged).

// real space: one block per (box, chunk of RES_TCH targets), as the near field
__global__ void __launch_bounds__(RES_T) k_ewald_real(DevTree T, int level, int ny, double alpha, double rc,
                                                      double* part) {
  __shared__ double ux[RES_SCH], uy[RES_SCH], uz[RES_SCH], uq[RES_SCH];
  __shared__ int uslot[RES_SCH];
  __shared__ int m_beg[27], m_pre[28];
  __shared__ double m_off[27][3];
  __shared__ double sm[32];
  const int node = T.level_start_d[level] + int(blockIdx.x) / ny, chunk = int(blockIdx.x) % ny;
  const int tb = T.node_begin[node];
  const int cnt = T.node_end[node] - tb;  // slots, empty ones carry q = 0
  double e = 0;
  if (cnt > chunk * RES_TCH) {
    const double b = level_box(T, level);
    const double rc2 = rc * rc;
    if (threadIdx.x < 27) {
      const int dir = threadIdx.x;
      const int j = dir == 13 ? node : T.col27[size_t(node) * 27 + dir];
      int beg = 0, n = 0;
      double off[3] = {0, 0, 0};
      if (j >= 0) {
        double ci[3], cj[3];
        node_center(T, node, ci);
        node_center(T, j, cj);
        for (int dd = 0; dd < 3; ++dd) off[dd] = -periodic_shift_d(ci[dd], cj[dd], T.L, b, b) * T.L;
        beg = T.node_begin[j];
        n = T.node_end[j] - beg;
      }
      m_beg[dir] = beg;
      m_pre[dir] = n;
      for (int dd = 0; dd < 3; ++dd) m_off[dir][dd] = off[dd];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int acc = 0;
      for (int src = 0; src < 27; ++src) {
        const int n = m_pre[src];
        m_pre[src] = acc;
        acc += n;
      }
      m_pre[27] = acc;
    }
    __syncthreads();
    const int total = m_pre[27];
    for (int t0 = chunk * RES_TCH; t0 < cnt; t0 += ny * RES_TCH) {
      const int nt = min(RES_TCH, cnt - t0);
      const int npad = nt <= 32 ? 32 : 64;
      const int nparts = RES_T / npad;
      const int it = threadIdx.x % npad, sp = threadIdx.x / npad;
      const bool act = it < nt;
      int tslot = -2;
      double tx = 0, ty = 0, tz = 0, tq = 0;
      if (act) {
        tslot = tb + t0 + it;
        tx = T.sx[tslot];
        ty = T.sy[tslot];
        tz = T.sz[tslot];
        tq = T.sq[tslot];
      }
      double et = 0;
      for (int u0 = 0; u0 < total; u0 += RES_SCH) {
        const int ns = min(RES_SCH, total - u0);
        __syncthreads();
        for (int t = threadIdx.x; t < ns; t += blockDim.x) {
          const int ei = u0 + t;
          int lo = 0, hi = 27;
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (m_pre[mid] <= ei) lo = mid;
            else hi = mid;
          }
          const int sl = m_beg[lo] + (ei - m_pre[lo]);
          ux[t] = T.sx[sl] + m_off[lo][0];
          uy[t] = T.sy[sl] + m_off[lo][1];
          uz[t] = T.sz[sl] + m_off[lo][2];
          uq[t] = T.sq[sl];
          uslot[t] = sl;
        }
        __syncthreads();
        if (act && tq != 0.0)
          for (int js = sp; js < ns; js += nparts) {
            const double dx = tx - ux[js], dy = ty - uy[js], dz = tz - uz[js];
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 < rc2 && uslot[js] != tslot && uq[js] != 0.0) {
              const double r = sqrt(r2);
              et += uq[js] * erfc(alpha * r) / r;
            }
          }
      }
      e += tq * et;
    }
  }
  double sum = block_sum(0.5 * e, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = sum;
}

// reciprocal space over the stored half grid kz <= 0 (kz < 0 stands for its
// mirror too)
__global__ void k_ewald_recip(const double2* __restrict__ S, int nk, double dk, double alpha, double* part) {
  __shared__ double sm[32];
  const int d = 2 * nk + 1;
  const long H = long(d) * d * (nk + 1);
  double e = 0;
  for (long k = long(blockIdx.x) * blockDim.x + threadIdx.x; k < H; k += long(gridDim.x) * blockDim.x) {
    const int ix = int(k % d), iy = int((k / d) % d), iz = int(k / (long(d) * d));
    const int mx = ix - nk, my = iy - nk, mz = iz - nk;
    if ((mx | my | mz) == 0) continue;
    const double k2 = dk * dk * double(mx * mx + my * my + mz * mz);
    const double2 v = S[k];
    e += (mz < 0 ? 2.0 : 1.0) * exp(-k2 / (4.0 * alpha * alpha)) / k2 * (v.x * v.x + v.y * v.y);
  }
  const double sum = block_sum(e, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = sum;
}

// rows 0 .. n unless a pass or an earlier call defined them
__global__ void k_zero_undefined(double2* rows, size_t n, const unsigned int* defined) {
  if (*defined) return;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    rows[i] = make_double2(0.0, 0.0);
}
__global__ void k_set_defined(unsigned int* counter, bool out, bool inc) {
  if (out) counter[14] = 1;
  if (inc) counter[15] = 1;
}

__global__ void k_sum(const double* part, int n, double* out) {
  __shared__ double sm[32];
  // eight loads in flight a thread: one at a time, the 2.6e5 near-field
  // partials of N = 1e6 took 31 us
  double e[8] = {};
  const int st = blockDim.x;
  for (int i = threadIdx.x; i < n; i += 8 * st) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i + u * st < n) e[u] += part[i + u * st];
  }
  double s = block_sum(((e[0] + e[1]) + (e[2] + e[3])) + ((e[4] + e[5]) + (e[6] + e[7])), sm);
  if (threadIdx.x == 0) *out = s;
}

// sum of q^2 over the slots: block b sums a grid-strided share into out[b]
// (one block gives the total in out[0])
__global__ void k_sum_q2(const double* sq, int n, double* out) {
  __shared__ double sm[32];
  double e = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) e += sq[i] * sq[i];
  double s = block_sum(e, sm);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

}  // namespace

// ---------------------------------------------------------------------------
// host side

constexpr int RES_NY_MAX = 8;  // the partials buffer holds this many near-field chunks per node

// target chunks per leaf in the near-field launch: enough for a full leaf
// with its slack (larger leaves loop over their chunks), at most the tuned cap
int DmkTree::res_chunks() const {
  return std::min(std::min(RES_NY_MAX, tune_.res_ny_max),
                  std::max(1, (n_per_leaf_ + opt_.leaf_slack + RES_TCH - 1) / RES_TCH));
}

void DmkTree::set_tuning(const Tuning& t) {
  Tuning c = t;
  // the mixed pass's exact int32 sums hold 16384 particles per split-K
  // chunk: an accumulator takes at most four slice products per K entry, top
  // digits lie in [-127, 127] and lower ones in [-128, 127], so one K entry
  // adds at most 2 127 128 + 2 128^2 = 65280, and two K entries per particle
  // give 2 16384 65280 < 2^31
  const int cap = opt_.precision == 1 ? 16384 : 1 << 20;
  c.ksplit = std::min(cap, std::max(256, c.ksplit));
  c.ksplit_root = std::min(cap, std::max(256, c.ksplit_root));
  c.inc_waves = std::min(64, std::max(1, c.inc_waves));
  c.res_ny_max = std::min(RES_NY_MAX, std::max(1, c.res_ny_max));
  tune_ = c;
}

double DmkTree::time_phase(int phase, int reps) {
  std::vector<float> ms;
  cudaEvent_t a, b;
  PDMK_CUDA(cudaEventCreate(&a));
  PDMK_CUDA(cudaEventCreate(&b));
  for (int r = 0; r < reps; ++r) {
    PDMK_CUDA(cudaStreamSynchronize(st_));
    PDMK_CUDA(cudaEventRecord(a, st_));
    if (phase == 0) {
      form_outgoing_pw();
    } else if (phase == 1) {
      form_incoming_pw();
    } else {
      ensure_packed();
      launch_res_energy();
    }
    PDMK_CUDA(cudaEventRecord(b, st_));
    PDMK_CUDA(cudaEventSynchronize(b));
    float t = 0;
    PDMK_CUDA(cudaEventElapsedTime(&t, a, b));
    ms.push_back(t);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  std::sort(ms.begin(), ms.end());
  return ms.empty() ? 0.0 : double(ms[ms.size() / 2]);
}

size_t DmkTree::partials_needed() const {
  const DevTree& D = dev_;
  size_t need = 8192;
  long n_pw = D.pw_hi >= D.pw_lo ? long(D.level_start[D.pw_hi + 1]) - D.level_start[D.pw_lo] : 0;
  long ktiles = (D.H + TPB - 1) / TPB;
  need = std::max<size_t>(need, size_t(n_pw) * ktiles + 2 * size_t(n_pw) + 64);
  // cube-tiled incoming: at most one cube per 8 expansion boxes
  need = std::max<size_t>(need, size_t((D.H + INC_KT - 1) / INC_KT) * size_t(n_pw / 8 + 1) + 2 * size_t(n_pw) + 64);
  need = std::max<size_t>(need, size_t(D.n_nodes) * RES_NY_MAX + 64);
  return need;
}

void DmkTree::ensure_packed() {
  // only accepted moves put particles into the overflow pool: a tree without
  // moves since its build or last pack needs no device round trip
  if (!moved_ && !captured_moves_) return;
  int pn = 0;
  PDMK_CUDA(cudaMemcpyAsync(&pn, dev_.pool_n, 4, cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  if (pn > 0) repack(opt_.leaf_slack);
  moved_ = false;
}

// A tree's rows are zero until a pass forms them. Clearing them in the build
// wrote every row twice (4.5 GB, 0.7 ms at N = 1e6 and 9 digits), so it waits
// for a call that reads a row no pass has formed. The device's own flags
// decide, so that a captured call does not clear formed rows when it is
// replayed.
void DmkTree::ensure_rows(bool out, bool inc) {
  out = out && !out_defined_;
  inc = inc && !inc_defined_;
  if (!out && !inc) return;
  const DevTree& D = dev_;
  const long n_pw = D.pw_hi >= D.pw_lo ? long(D.level_start[D.pw_hi + 1]) - D.level_start[D.pw_lo] : 0;
  const size_t n = size_t(std::max<long>(n_pw, 1)) * D.H;
  if (out) k_zero_undefined<<<1184, 256, 0, st_>>>(D.out, n, D.counter + 14);
  if (inc) k_zero_undefined<<<1184, 256, 0, st_>>>(D.inc, n, D.counter + 15);
  k_set_defined<<<1, 1, 0, st_>>>(D.counter, out, inc);
  PDMK_LAUNCH_CHECK();
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  PDMK_CUDA(cudaStreamIsCapturing(st_, &cs));
  if (cs != cudaStreamCaptureStatusNone) return;  // nothing ran yet
  out_defined_ |= out;
  inc_defined_ |= inc;
}

void DmkTree::form_outgoing_pw() {
  ensure_packed();
  ensure_dense();
  DevTree& D = dev_;
  const int n_all = int(N_);
  const bool mixed = opt_.precision == 1;
  CUtensorMap tmap_root{}, tmap_box{};
  if (mixed) {
    if (!d_mix_) {
      d_mix_ = static_cast<double*>(alloc(sizeof(double) * 2));
      PDMK_CUDA(cudaMemsetAsync(d_mix_, 0, sizeof(double) * 2, st_));
    }
    if (!qmax_ready_) {
      launch_absmax(dense_ + 3 * dense_stride_, n_all, d_mix_, st_);
      qmax_ready_ = true;
    }
    make_coord_map(&tmap_root, dense_, int(dense_stride_), mixed_chunk(D.n_window));
    make_coord_map(&tmap_box, dense_, int(dense_stride_), mixed_chunk(D.n_diff));
  }
  int* d_mix_err = mixed ? reinterpret_cast<int*>(d_mix_ + 1) : nullptr;
  auto get = [&](size_t bytes) {
    void* p = nullptr;
    PDMK_CUDA(cudaMallocAsync(&p, bytes + 16, st_));
    return static_cast<unsigned char*>(p);
  };
  // a pass's items, split entries and chunk list in one block
  struct Lists {
    unsigned char* block;
    PwItem* items;
    PwSplit* split;
    int2* chunks;
    int* next;  // the mixed pass's tile counter
  };
  auto get_lists = [&](int n_items, int n_split, int n_chunks) {
    Lists l;
    l.block = get(sizeof(PwItem) * size_t(n_items) + sizeof(PwSplit) * size_t(n_split) + sizeof(int2) * size_t(n_chunks + 1));
    l.items = reinterpret_cast<PwItem*>(l.block);
    l.split = reinterpret_cast<PwSplit*>(l.items + n_items);
    l.chunks = reinterpret_cast<int2*>(l.split + n_split);
    l.next = reinterpret_cast<int*>(l.chunks + n_chunks);
    return l;
  };
  auto contract = [&](int nk, const CUtensorMap& tmap, const Lists& l, int n_items, int n_chunks, cudaStream_t st) {
    if (mixed) dispatch_mixed(nk, tmap, l.items, n_items, l.chunks, n_chunks, l.next, d_mix_, d_mix_err, st);
    else dispatch_nudft(nk, l.items, n_items, dense_, dense_stride_, st);
  };
  if (!aux_) {
    aux_ = take_stream(&aux_device_);
    PDMK_CUDA(cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming));
    PDMK_CUDA(cudaEventCreateWithFlags(&ev_join_, cudaEventDisableTiming));
  }
  // A small system would leave most SMs idle behind a few blocks that each
  // walk all particles: its items are cut until they give one wave of blocks
  // (the root, which runs beside the boxes: half a wave), not below 64
  // particles. Finer cuts cost more than they fill: a partial row's way to
  // memory and back is worth 45 particles. Outgoing pass in us, uncut / half and
  // one wave / two and two waves: N = 1e3 (6 digits) 172 / 63 / 61, 5e3 (9
  // digits) 170 / 118 / 186, 2e4 223 / 217 / 321, 5e4 437 / 441 / 560, 128e3 (3
  // digits) 218 / 172 / 160.
  auto fill_split = [&](int split, long particles, int tiles, int blocks) {
    const long want = std::max(1, (blocks + tiles - 1) / tiles);  // items
    return int(std::min<long>(split, std::max<long>(64, (particles + want - 1) / want)));
  };
  auto shape = [&](int nk, int ksplit) {
    return PlanShape{ksplit, mixed ? mixed_chunk(nk) : 1, mixed ? long(mixed_table_bytes(nk)) : 0L};
  };
  const long pw_levels = std::max(0, D.pw_hi - D.pw_lo + 1);
  const PlanShape root_shape = shape(
      D.n_window, mixed ? tune_.ksplit_root : fill_split(tune_.ksplit_root, n_all, nudft_tiles(D.n_window), 148));
  const PlanShape box_shape = shape(
      D.n_diff, mixed ? tune_.ksplit : fill_split(tune_.ksplit, pw_levels * n_all, nudft_tiles(D.n_diff), 296));

  // the boxes' totals, counted before the root pass takes the device
  const bool lists = !box_lists_ready_;
  const size_t state_bytes = (sizeof(PlanState) + 15) & ~size_t(15);
  unsigned char* d_plan = get(state_bytes + sizeof(int) * 3 * size_t(plan_blocks(D.n_nodes)));
  PlanState* d_state = reinterpret_cast<PlanState*>(d_plan);
  int* d_blk = reinterpret_cast<int*>(d_plan + state_bytes);
  PDMK_CUDA(cudaMemsetAsync(d_state, 0, sizeof(PlanState), st_));
  launch_plan_count(D, box_shape, lists, d_state, d_blk, st_);

  // Root pass on the second stream: the root (node 0, all particles) needs no
  // totals, so it runs while they travel. Its allocations are made on the
  // tree's stream before the fork event.
  const int n_root = std::max(1, (n_all + root_shape.ksplit - 1) / root_shape.ksplit);
  const int root_full = (root_shape.ksplit + root_shape.kcp - 1) / root_shape.kcp;
  const int n_root_chunks = !mixed ? 0
                                   : (n_root - 1) * root_full +
                                         (n_all - (n_root - 1) * root_shape.ksplit + root_shape.kcp - 1) / root_shape.kcp;
  double2* part_r = reinterpret_cast<double2*>(get(sizeof(double2) * size_t(n_root) * D.Hw));
  unsigned char* tab_r = mixed ? get(size_t(n_root_chunks) * root_shape.tab_bytes) : nullptr;
  const Lists root = get_lists(n_root, 1, n_root_chunks);
  launch_plan_root(D, root_shape, n_all, n_root, n_root_chunks, part_r, tab_r, root.items, root.chunks, root.split, root.next, st_);
  PDMK_CUDA(cudaEventRecord(ev_fork_, st_));
  PDMK_CUDA(cudaStreamWaitEvent(aux_, ev_fork_, 0));
  contract(D.n_window, tmap_root, root, n_root, n_root_chunks, aux_);
  launch_reduce_chunks(part_r, root.split, 1, n_root, D.Hw, aux_);
  PDMK_CUDA(cudaEventRecord(ev_join_, aux_));

  PlanTotals t;
  PDMK_CUDA(cudaMemcpyAsync(&t, &d_state->t, sizeof(t), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  double2* part_b = reinterpret_cast<double2*>(get(sizeof(double2) * size_t(t.n_split_items) * D.H));
  unsigned char* tab_b = mixed ? get(size_t(t.n_chunks) * box_shape.tab_bytes) : nullptr;
  const Lists box = get_lists(t.n_items, t.n_split, t.n_chunks);
  launch_plan_items(D, box_shape, node_dense_, d_state, part_b, tab_b, box.items, box.chunks, box.split, box.next, st_);
  time_begin(3);
  contract(D.n_diff, tmap_box, box, t.n_items, t.n_chunks, st_);
  time_end(3);
  launch_reduce_chunks(part_b, box.split, t.n_split, t.n_split_items, D.H, st_);
  out_defined_ = true;
  out_formed_ = true;
  if (lists) fill_box_lists(t, d_blk);
  // the root pass's buffers are released after it joins the tree's stream
  PDMK_CUDA(cudaStreamWaitEvent(st_, ev_join_, 0));
  for (void* p : {static_cast<void*>(root.block), static_cast<void*>(tab_r), static_cast<void*>(part_r),
                  static_cast<void*>(box.block), static_cast<void*>(tab_b), static_cast<void*>(part_b),
                  static_cast<void*>(d_plan)})
    if (p) PDMK_CUDA(cudaFreeAsync(p, st_));
  diff_cached_ = false;
}

void DmkTree::prepare_box_lists() {
  if (box_lists_ready_) return;
  void* d_plan = nullptr;
  const size_t state_bytes = (sizeof(PlanState) + 15) & ~size_t(15);
  PDMK_CUDA(cudaMallocAsync(&d_plan, state_bytes + sizeof(int) * 3 * size_t(plan_blocks(dev_.n_nodes)), st_));
  PlanState* state = static_cast<PlanState*>(d_plan);
  int* blk = reinterpret_cast<int*>(static_cast<unsigned char*>(d_plan) + state_bytes);
  PDMK_CUDA(cudaMemsetAsync(state, 0, sizeof(PlanState), st_));
  launch_plan_count(dev_, PlanShape{1 << 30, 1, 0}, true, state, blk, st_);
  PlanTotals t;
  PDMK_CUDA(cudaMemcpyAsync(&t, &state->t, sizeof(t), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  fill_box_lists(t, blk);
  PDMK_CUDA(cudaFreeAsync(d_plan, st_));
}

// the lists behind counted totals (blk: the per-block counts)
void DmkTree::fill_box_lists(const PlanTotals& t, const int* blk) {
  DevTree& D = dev_;
  n_nonleaf_ = t.n_nonleaf;
  n_leaves_ = t.n_leaves;
  n_cubes_ = t.n_cubes;
  d_nonleaf_ = static_cast<int*>(alloc(sizeof(int) * size_t(n_nonleaf_ + n_leaves_ + n_cubes_ + 1)));
  d_leaves_ = d_nonleaf_ + n_nonleaf_;
  d_cubes_ = d_leaves_ + n_leaves_;
  launch_plan_lists(D, blk, d_nonleaf_, d_leaves_, d_cubes_, st_);
  // sum(q^2) for the window self term: 592 block partials (64 took 38 us at
  // N = 1e6), then a fixed-order sum
  k_sum_q2<<<592, 256, 0, st_>>>(D.sq, D.n_slots, D.partials);
  PDMK_LAUNCH_CHECK();
  k_sum<<<1, 1024, 0, st_>>>(D.partials, 592, d_scalars_ + 4);
  PDMK_LAUNCH_CHECK();
  box_lists_ready_ = true;
}

void DmkTree::run_incoming(bool write_inc) {
  ensure_packed();
  prepare_box_lists();
  DevTree& D = dev_;
  ensure_rows(true, !write_inc);
  if (n_nonleaf_ == 0) {
    PDMK_CUDA(cudaMemsetAsync(d_scalars_ + 1, 0, sizeof(double), st_));
    return;
  }
  const int ktiles = (D.H + TPB - 1) / TPB;
  const size_t n_part = std::max(size_t(ktiles) * n_nonleaf_, size_t((D.H + INC_KT - 1) / INC_KT) * n_cubes_);
  double* part = D.partials;
  double* q2 = D.partials + n_part;
  k_box_q2<<<unsigned(n_nonleaf_), TPB, 0, st_>>>(D, d_nonleaf_, q2);
  PDMK_LAUNCH_CHECK();
  if (write_inc) {
    // about inc_waves waves of blocks (counted at two per SM), each walking a
    // strided set of tiles
    const int slots = inc_slots();
    inc_defined_ = true;  // the non-leaf boxes' rows; a leaf's row is read by nothing
    if (n_cubes_ > 0) launch_incoming(D, d_cubes_, n_cubes_, slots, part, nullptr, st_);
    k_diff_finish_cube<<<1, 1024, 0, st_>>>(D, d_cubes_, n_cubes_, slots, part, d_nonleaf_, n_nonleaf_, q2, d_Cl_,
                                            d_Sl_, d_scalars_ + 1);
    PDMK_LAUNCH_CHECK();
  } else {
    k_tridot<<<unsigned(ktiles * n_nonleaf_), TPB, 0, st_>>>(D, d_nonleaf_, n_nonleaf_, part);
    PDMK_LAUNCH_CHECK();
    k_diff_finish<<<1, 1024, 0, st_>>>(D, d_nonleaf_, n_nonleaf_, ktiles, part, q2, d_Cl_, d_Sl_, d_scalars_ + 1);
    PDMK_LAUNCH_CHECK();
  }
}

int DmkTree::inc_slots() const {
  const int kt = (dev_.H + INC_KT - 1) / INC_KT;
  const int nc = std::max(n_cubes_, 1);
  return std::max(1, std::min(kt, (tune_.inc_waves * 2 * 148 + nc - 1) / nc));
}

void launch_incoming_set(int n_diff, const DevTree* trees, const SequenceRows* rows, int n_trees, int blocks,
                         cudaStream_t st) {
  if (blocks == 0) return;
  switch (n_diff) {
    case 6: launch_incoming_set_nk<6>(trees, rows, n_trees, blocks, st); break;
    case 12: launch_incoming_set_nk<12>(trees, rows, n_trees, blocks, st); break;
    case 19: launch_incoming_set_nk<19>(trees, rows, n_trees, blocks, st); break;
    case 26: launch_incoming_set_nk<26>(trees, rows, n_trees, blocks, st); break;
    default: throw std::invalid_argument("incoming pass: unsupported mode count");
  }
}

// The incoming rows next to outgoing rows that changed (touched[expansion
// node] != 0), after a sequence of moves. The partial energies go unused.
void DmkTree::launch_incoming_touched(const int* touched) {
  if (n_cubes_ > 0) launch_incoming(dev_, d_cubes_, n_cubes_, inc_slots(), dev_.partials, touched, st_);
}

void DmkTree::form_incoming_pw() {
  run_incoming(true);
  diff_cached_ = true;
  // outgoing rows that no pass formed hold the accepted moves alone, and emptied
  // boxes among them are not zero, as the recomputation takes them to be
  inc_formed_ = out_formed_;
}

void DmkTree::launch_window_energy() {
  prepare_box_lists();
  DevTree& D = dev_;
  const double pi = 3.14159265358979323846;
  double scale = 1 / (2 * std::pow(2 * pi, 3)) * std::pow(D.delta_k[0], 3);
  k_window<<<1, 1024, 0, st_>>>(D, scale, d_scalars_ + 4, ps_.psi0_0, 2 * D.boxsize[2] * ps_.C0, d_scalars_ + 0);
  PDMK_LAUNCH_CHECK();
}

double DmkTree::eval_window_energy() {
  launch_window_energy();
  double e;
  PDMK_CUDA(cudaMemcpyAsync(&e, d_scalars_ + 0, sizeof(double), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  return e;
}

double DmkTree::eval_diff_energy() {
  ensure_packed();
  if (!diff_cached_) run_incoming(false);
  double e;
  PDMK_CUDA(cudaMemcpyAsync(&e, d_scalars_ + 1, sizeof(double), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  return e;
}

void DmkTree::launch_res_energy() {
  prepare_box_lists();
  DevTree& D = dev_;
  if (n_leaves_ > 0) {
    auto pick = [&](auto minb) {
      constexpr int B = decltype(minb)::value;
      return D.n_poly == 7 ? k_residual<7, B> : D.n_poly == 13 ? k_residual<13, B> : D.n_poly == 19 ? k_residual<19, B>
                                                                                                    : k_residual<25, B>;
    };
    // between the two measured fillings
    auto kern = N_ >= 40 * long(n_leaves_) ? pick(std::integral_constant<int, 7>{}) : pick(std::integral_constant<int, 9>{});
    const int ny = res_chunks();
    kern<<<unsigned(n_leaves_ * ny), RES_T, 0, st_>>>(D, d_leaves_, ny, D.partials);
    PDMK_LAUNCH_CHECK();
    k_sum<<<1, 1024, 0, st_>>>(D.partials, n_leaves_ * ny, d_scalars_ + 2);
    PDMK_LAUNCH_CHECK();
  } else {
    PDMK_CUDA(cudaMemsetAsync(d_scalars_ + 2, 0, sizeof(double), st_));
  }
}

double DmkTree::eval_res_energy() {
  ensure_packed();
  launch_res_energy();
  double e = 0;
  PDMK_CUDA(cudaMemcpyAsync(&e, d_scalars_ + 2, sizeof(double), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  return e;
}

int DmkTree::check_mixed_error() {
  if (!d_mix_) return 0;
  int e = 0;
  PDMK_CUDA(cudaMemcpyAsync(&e, d_mix_ + 1, sizeof(int), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  return e;
}

EnergyParts DmkTree::eval_energy() {
  // per-box charge sums and the near field read particles from the slot
  // ranges: fold any overflow-pool arrivals back into them first. The three
  // parts are enqueued back to back and read with one synchronisation.
  ensure_packed();
  launch_window_energy();
  if (!diff_cached_) run_incoming(false);
  launch_res_energy();
  double e[3];
  int mix_err = 0;
  PDMK_CUDA(cudaMemcpyAsync(e, d_scalars_, sizeof(e), cudaMemcpyDeviceToHost, st_));
  if (d_mix_) PDMK_CUDA(cudaMemcpyAsync(&mix_err, d_mix_ + 1, sizeof(int), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  if (mix_err) throw DeviceError("mixed-precision outgoing pass: a pipeline wait gave up");
  EnergyParts p;
  p.window = e[0];
  p.diff = e[1];
  p.res = e[2];
  return p;
}

// FP64 Ewald energy of the current particles (comparator; s = 5: erfc(5) and
// exp(-25) put the truncation near 1e-12 relative). The real-space cut-off is
// the box size of level 2, or of level 3 when that level is complete and the
// system is large; the k cube then needs 32 or 64 modes per axis half.
double DmkTree::ewald_energy(double* parts) {
  ensure_packed();
  ensure_dense();
  DevTree& D = dev_;
  const double s = 5.0, pi = 3.14159265358979323846;
  const bool l3 = D.max_depth > 4 && D.level_start[4] - D.level_start[3] == 512 && D.n_slots > 300000;
  const int le = l3 ? 3 : 2;
  const int nk = l3 ? 64 : 32;
  const double rc = std::ldexp(L_, -le), alpha = s / rc, dk = 2 * pi / L_;
  const int nbox = D.level_start[le + 1] - D.level_start[le];
  // chunks of targets per box: enough for the fullest box of the level
  std::vector<int> nb(nbox), ne(nbox);
  PDMK_CUDA(cudaMemcpyAsync(nb.data(), D.node_begin + D.level_start[le], 4 * nbox, cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaMemcpyAsync(ne.data(), D.node_end + D.level_start[le], 4 * nbox, cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  int maxc = 1;
  for (int b = 0; b < nbox; ++b) maxc = std::max(maxc, ne[b] - nb[b]);
  const int ny = (maxc + RES_TCH - 1) / RES_TCH;
  // structure factor by the NUDFT over all slots, split in chunks
  const int Hs = (2 * nk + 1) * (2 * nk + 1) * (nk + 1);
  const int n_all = int(N_);
  const int kspl = std::max(4096, (n_all + 295) / 296);
  const int nch = std::max(1, (n_all + kspl - 1) / kspl);
  std::vector<PwItem> wl;
  for (int c = 0; c < nch; ++c) {
    PwItem w{};
    w.cx = w.cy = w.cz = 0.5 * L_;
    w.dk = dk;
    w.M = 3;  // exp(-i k L/2) = (-1)^m: the root's decentring
    w.s_begin = c * kspl;
    w.s_end = std::min(n_all, (c + 1) * kspl);
    wl.push_back(w);
  }
  double2* part = nullptr;
  double2* S = nullptr;
  PwItem* d_work = nullptr;
  const int nblk_real = nbox * ny, nblk_rec = 1024;
  double* sums = nullptr;
  PDMK_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&part), sizeof(double2) * size_t(Hs) * nch, st_));
  PDMK_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&S), sizeof(double2) * size_t(Hs), st_));
  PDMK_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&sums), sizeof(double) * (nblk_real + nblk_rec + 8), st_));
  for (size_t i = 0; i < wl.size(); ++i) wl[i].out = part + i * size_t(Hs);
  PDMK_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&d_work), sizeof(PwItem) * wl.size(), st_));
  PDMK_CUDA(cudaMemcpyAsync(d_work, wl.data(), sizeof(PwItem) * wl.size(), cudaMemcpyHostToDevice, st_));
  dispatch_nudft(nk, d_work, int(wl.size()), dense_, dense_stride_, st_);
  {
    PwSplit* d_split;
    const PwSplit all{0, nch, S};
    PDMK_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&d_split), sizeof(PwSplit), st_));
    PDMK_CUDA(cudaMemcpyAsync(d_split, &all, sizeof(PwSplit), cudaMemcpyHostToDevice, st_));
    launch_reduce_chunks(part, d_split, 1, nch, Hs, st_);
    PDMK_CUDA(cudaFreeAsync(d_split, st_));
  }
  k_ewald_recip<<<unsigned(nblk_rec), TPB, 0, st_>>>(S, nk, dk, alpha, sums + nblk_real);
  PDMK_LAUNCH_CHECK();
  k_ewald_real<<<unsigned(nblk_real), RES_T, 0, st_>>>(D, le, ny, alpha, rc, sums);
  PDMK_LAUNCH_CHECK();
  k_sum<<<1, 1024, 0, st_>>>(sums, nblk_real, sums + nblk_real + nblk_rec);
  PDMK_LAUNCH_CHECK();
  k_sum<<<1, 1024, 0, st_>>>(sums + nblk_real, nblk_rec, sums + nblk_real + nblk_rec + 1);
  PDMK_LAUNCH_CHECK();
  k_sum_q2<<<1, 1024, 0, st_>>>(D.sq, D.n_slots, sums + nblk_real + nblk_rec + 2);
  PDMK_LAUNCH_CHECK();
  double r3[3];
  PDMK_CUDA(cudaMemcpyAsync(r3, sums + nblk_real + nblk_rec, sizeof(r3), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaFreeAsync(part, st_));
  PDMK_CUDA(cudaFreeAsync(S, st_));
  PDMK_CUDA(cudaFreeAsync(d_work, st_));
  PDMK_CUDA(cudaFreeAsync(sums, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  const double e_real = r3[0];
  const double e_rec = 2 * pi / (L_ * L_ * L_) * r3[1];
  const double e_self = -alpha / std::sqrt(pi) * r3[2];
  if (parts) {
    parts[0] = e_real;
    parts[1] = e_rec;
    parts[2] = e_self;
  }
  return e_real + e_rec + e_self;
}

}  // namespace pdmk
