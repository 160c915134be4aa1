// Single-particle energy shift, accept-and-update, and the device-side
// Metropolis loop (FP64).
//
// Reference counterparts: eval_shift_energy and its window / difference /
// residual parts (src/energy_shift.cpp:18-302), locate_particle
// (src/tree.cpp:204-236), form_outgoing_pw_single (src/planewave.cpp:157-181)
// and update_shift (src/tree.cpp:447-597).
//
// One trial move runs as: k_shift (grid-wide partial sums, and one block that
// lists the expansion vectors an accepted move changes; the last block finishes
// dE and the Metropolis test and writes the Proposal record), then k_update (one
// read-modify-write per touched vector, target and origin contributions
// merged; block 0 also commits the particle membership). Both kernels read
// the Proposal record, so the sequence is stream-ordered and can be captured
// in a CUDA graph. Per-move latency is what bounds Monte Carlo throughput,
// so the kernels avoid dependent global loads: box coordinates along both
// paths come from the particle's grid key, the 27 minimum-image candidates
// and the two paths are resolved by the lanes of one warp in parallel.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "tree.hpp"

namespace pdmk {
namespace {

constexpr int SH_T = 256;
constexpr int MAXLV = MAX_LEVELS;

__device__ inline bool bm_get(const uint32_t* bm, uint64_t cell) { return (bm[cell >> 5] >> (cell & 31)) & 1u; }

__device__ inline int bm_rank(const DevTree& T, int level, uint64_t cell) {
  uint32_t w = T.bm_d[level][cell >> 5];
  return T.wprefix_d[level][cell >> 5] + __popc(w & ((1u << (cell & 31)) - 1u));
}

__device__ inline double center_of(double L, int l, int X) {
  double scale = ldexp(1.0, -l);
  return L * (double(X) * scale + 0.5 * scale);
}

__device__ inline int periodic_shift_d(double xi, double xj, double L, double bi, double bj) {
  if (xi < bi && xj > (L - bj)) return 1;
  if (xi > (L - bi) && xj < bj) return -1;
  return 0;
}


// Phase tables exp(-i m dk_l x) per axis for one point on its path. Layout:
// root axes (3 x dw), then levels 2, 3, ... (3 x dd each). The accessors
// compute addresses, so no pointer array is indexed at run time.
struct Tables {
  struct Axes {
    double2* b;
    int stride;
    __device__ double2* operator[](int ax) const { return b + ax * stride; }
  };
  struct Levels {
    double2* b;
    int dw, dd;
    __device__ Axes operator[](int l) const { return Axes{b + 3 * dw + (l - 2) * 3 * dd, dd}; }
  };
  Axes root;
  Levels lev;
};

__device__ inline void alloc_tables(double2* sm, const DevTree& T, Tables& tb) {
  tb.root = Tables::Axes{sm, 2 * T.n_window + 1};
  tb.lev = Tables::Levels{sm, 2 * T.n_window + 1, 2 * T.n_diff + 1};
}

struct Header {
  int i_orig, slot;
  double q;
  double xo[3], xt[3];
  double dr;
  int depth_o, depth_t;
  int path_o[MAXLV], path_t[MAXLV];
  int Xo[MAXLV][3], Xt[MAXLV][3];  // integer box coordinates along each path
  double d2;                       // k_mc_long: squared length of the displacement
};

// Tables of one point on its path for levels 2..lmax, one entry per thread
// (threads t0, t0 + nthr, ...): e^{-i m dk_l (x - c_l)} with the box-centred
// phase and the exact decentring root of unity, times q on the z axis. Every
// entry is its own sincos, so the table costs one sincos latency instead of
// a chain of recurrence steps.
__device__ void build_tables(const DevTree& T, const double* x, double q, const int (*X)[3], int lmax,
                             const Tables& tb, int t0, int nthr) {
  const int nw = T.n_window, nd = T.n_diff;
  const int root_n = 2 * (2 * nw + 1) + (nw + 1);
  const int lev_n = 2 * (2 * nd + 1) + (nd + 1);
  const int nlev = lmax >= 2 ? lmax - 1 : 0;
  const int total = root_n + nlev * lev_n;
  for (int e = t0; e < total; e += nthr) {
    int slot, rem;
    if (e < root_n) {
      slot = 0;
      rem = e;
    } else {
      slot = 1 + (e - root_n) / lev_n;
      rem = (e - root_n) % lev_n;
    }
    const int n = slot == 0 ? nw : nd;
    const int w = 2 * n + 1;
    const int axis = rem < w ? 0 : (rem < 2 * w ? 1 : 2);
    const int t = rem - axis * w;
    const int m = t - n;
    double xr, dk;
    int dec;
    double2* dst;
    if (slot == 0) {
      xr = x[axis] - 0.5 * T.L;
      dk = T.delta_k[0];
      dec = 3;
      dst = tb.root[axis];
    } else {
      const int l = slot + 1, Xa = X[l][axis];
      xr = x[axis] - center_of(T.L, l, Xa);
      dk = level_dk(T, l);
      dec = 2 * Xa + 1;
      dst = tb.lev[l][axis];
    }
    const double th = dk * xr;
    double sn, cs;
    sincos(-double(m) * th, &sn, &cs);
    const double sc = axis == 2 ? q : 1.0;
    dst[t] = cmul(make_double2(cs * sc, sn * sc), root6(-dec * m));
  }
}

template <class A>
__device__ inline double2 phase_at(const A& ax, int k, int d) {
  int ix = k % d, iy = (k / d) % d, iz = k / (d * d);
  return cmul(ax[2][iz], cmul(ax[1][iy], ax[0][ix]));
}

// Resolve a proposal with the first warp: particle and positions (every lane
// loads the same words), my_mod wrap, the minimum-image old-new distance
// (one image per lane, src/energy_shift.cpp:30-41) and both leaf paths
// (lanes 0-15 the target, 16-31 the origin, one level per lane, from the
// refinement bitmaps: the reference's locate_particle, src/tree.cpp:204-236).
// Loads of data that other blocks of a persistent kernel write (CG = true)
// bypass L1, which is not coherent across SMs.
template <bool CG, class V>
__device__ inline V ldm(const V* p) {
  if constexpr (CG) return __ldcg(p);
  else return *p;
}

// A particle's slot, position and charge loaded ahead of its resolve (s < 0:
// nothing loaded).
struct Preload {
  int s;
  double x, y, z, q;
};

template <bool CG = false>
__device__ inline void resolve_by_warp(const DevTree& T, int i, const double* disp, Header& h, const Preload* pre = nullptr) {
  {
    const int lane = threadIdx.x & 31;
    const bool have = pre && pre->s >= 0;
    const int s = have ? pre->s : ldm<CG>(T.orig_slot + i);
    double xo[3], q;
    if (have) {
      xo[0] = pre->x;
      xo[1] = pre->y;
      xo[2] = pre->z;
      q = pre->q;
    } else if (s < T.n_slots) {
      xo[0] = ldm<CG>(T.sx + s);
      xo[1] = ldm<CG>(T.sy + s);
      xo[2] = ldm<CG>(T.sz + s);
      q = ldm<CG>(T.sq + s);
    } else {
      const int p = s - T.n_slots;
      xo[0] = ldm<CG>(T.px + p);
      xo[1] = ldm<CG>(T.py + p);
      xo[2] = ldm<CG>(T.pz + p);
      q = ldm<CG>(T.pq + p);
    }
    const double L = T.L;
    const double d0 = disp[0], d1 = disp[1], d2 = disp[2];
    const double xt[3] = {wrap_mod(xo[0] + d0, L), wrap_mod(xo[1] + d1, L), wrap_mod(xo[2] + d2, L)};
    double dr = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    if (lane < 27) {
      const int mx = lane % 3 - 1, my = (lane / 3) % 3 - 1, mz = lane / 9 - 1;
      const double ax = xt[0] - (xo[0] + mx * L), ay = xt[1] - (xo[1] + my * L), az = xt[2] - (xo[2] + mz * L);
      dr = fmin(dr, sqrt(ax * ax + ay * ay + az * az));
    }
    for (int o = 16; o > 0; o >>= 1) dr = fmin(dr, __shfl_xor_sync(0xffffffffu, dr, o));
    const int half = lane >> 4, l = lane & 15;
    const double* p = half == 0 ? xt : xo;
    const uint32_t g[3] = {grid_coord(p[0], L), grid_coord(p[1], L), grid_coord(p[2], L)};
    const uint64_t key = morton3(g[0], g[1], g[2]);
    bool is_leaf = false;
    int node = -1;
    if (l < T.max_depth) {
      const uint64_t cell = l == 0 ? 0 : key >> (3 * (KEY_BITS - l));
      const bool exists = l <= 1 || bm_get(T.bm_d[l - 1], cell >> 3);
      if (exists) {
        node = l == 0 ? 0
                      : (l == 1 ? 1 + int(cell) : T.level_start_d[l] + 8 * bm_rank(T, l - 1, cell >> 3) + int(cell & 7));
        is_leaf = !(l <= T.maxref && bm_get(T.bm_d[l], cell));
      }
    }
    const unsigned leaves = (__ballot_sync(0xffffffffu, is_leaf) >> (16 * half)) & 0xffffu;
    const int leaf_level = __ffs(leaves) - 1;
    if (l <= leaf_level) {
      int* path = half == 0 ? h.path_t : h.path_o;
      int(*X)[3] = half == 0 ? h.Xt : h.Xo;
      path[l] = node;
      for (int a = 0; a < 3; ++a) X[l][a] = int(g[a] >> (KEY_BITS - l));
    }
    if (lane == 0) {
      h.i_orig = i;
      h.slot = s;
      h.q = q;
      for (int a = 0; a < 3; ++a) {
        h.xo[a] = xo[a];
        h.xt[a] = xt[a];
      }
      h.dr = dr;
      h.depth_t = leaf_level + 1;
    }
    if (lane == 16) h.depth_o = leaf_level + 1;
  }
}

template <bool CG = false>
__device__ void resolve(const DevTree& T, int i, const double* disp, Header& h, const Preload* pre = nullptr) {
  if (threadIdx.x < 32) resolve_by_warp<CG>(T, i, disp, h, pre);
  __syncthreads();
}

// q * sum_{j in N(leaf)} q_j res(|x - x_j|; bs_leaf), masked r^2 in (eps, b^2)
// (eval_shift_energy_res_vec + direct_eval, src/energy_shift.cpp:233-302).
// Source metadata is fetched in parallel, then all threads share the pairs.
template <int NP>
__device__ double residual_sum(const DevTree& T, const ResidualPoly<NP>& poly, int leaf, int l, const int* Xl,
                               const double* x) {
  const double b = level_box(T, l);
  const double b2 = b * b;
  const double eps = 2.220446049250313e-16;
  __shared__ int m_beg[36], m_cnt[36], m_pre[37], m_lvl[36];
  __shared__ unsigned long long m_pfx[36];
  __shared__ double m_off[36][3];
  if (threadIdx.x < 36) {
    const int src = threadIdx.x;
    int j = -1;
    if (src == 0) j = leaf;
    else if (src <= 27) j = (src - 1 == 13) ? -1 : T.col27[size_t(leaf) * 27 + (src - 1)];
    else j = T.coarse8[size_t(leaf) * 8 + (src - 28)];
    int beg = 0, cnt = 0, lj = 0;
    unsigned long long pj = 0;
    double off[3] = {0, 0, 0};
    if (j >= 0) {
      lj = T.node_level[j];
      pj = T.node_prefix[j];
      const int ch = T.node_child0[j];
      beg = T.node_begin[j];
      const int end = ch < 0 ? beg + T.leaf_count[j] : T.node_end[j];
      cnt = end - beg;
      const double bj = level_box(T, lj);
      const int Xj[3] = {int(compact3(pj)), int(compact3(pj >> 1)), int(compact3(pj >> 2))};
      for (int d = 0; d < 3; ++d)
        off[d] = -periodic_shift_d(center_of(T.L, l, Xl[d]), center_of(T.L, lj, Xj[d]), T.L, b, bj) * T.L;
    }
    m_beg[src] = beg;
    m_cnt[src] = j >= 0 ? cnt : -1;
    m_lvl[src] = lj;
    m_pfx[src] = pj;
    for (int d = 0; d < 3; ++d) m_off[src][d] = off[d];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int src = 0; src < 36; ++src) {
      m_pre[src] = s;
      s += max(m_cnt[src], 0);
    }
    m_pre[36] = s;
  }
  __syncthreads();
  const int total = m_pre[36];
  double acc = 0;
  int src = 0;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    while (e >= m_pre[src + 1]) ++src;
    const int s = m_beg[src] + (e - m_pre[src]);
    const double dx = x[0] - (T.sx[s] + m_off[src][0]), dy = x[1] - (T.sy[s] + m_off[src][1]),
                 dz = x[2] - (T.sz[s] + m_off[src][2]);
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > eps && r2 < b2) acc += T.sq[s] * poly(sqrt(r2), b);
  }
  // arrivals parked in the overflow pool that belong to a source's subtree
  const int pn = *T.pool_n;
  for (int e = threadIdx.x; e < 36 * pn; e += blockDim.x) {
    const int sj = e / pn, p = e % pn;
    if (m_cnt[sj] < 0 || T.p_orig[p] < 0) continue;
    const int pl = T.p_leaf[p];
    const int ll = T.node_level[pl], lj = m_lvl[sj];
    if (ll < lj || (T.node_prefix[pl] >> (3 * (ll - lj))) != m_pfx[sj]) continue;
    const double dx = x[0] - (T.px[p] + m_off[sj][0]), dy = x[1] - (T.py[p] + m_off[sj][1]),
                 dz = x[2] - (T.pz[p] + m_off[sj][2]);
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > eps && r2 < b2) acc += T.pq[p] * poly(sqrt(r2), b);
  }
  return acc;
}

// sums of four values over the block, valid in thread 0
__device__ inline void block_sum4(double* v, double (*sm)[32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
  __syncthreads();
  if (lane == 0)
    for (int c = 0; c < 4; ++c) sm[c][warp] = v[c];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int c = 0; c < 4; ++c) {
      double s = 0;
      for (int w = 0; w < nw; ++w) s += sm[c][w];
      v[c] = s;
    }
  __syncthreads();
}

// as block_sum4, the sums in thread 0 only and no barrier after them (the
// caller's next barrier orders its use)
__device__ inline void block_sum4_t0(double* v, double (*sm)[32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
  __syncthreads();
  if (lane == 0)
    for (int c = 0; c < 4; ++c) sm[c][warp] = v[c];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int c = 0; c < 4; ++c) {
      double s = 0;
      for (int w = 0; w < nw; ++w) s += sm[c][w];
      v[c] = s;
    }
}

// slot s of a path level: 0 own outgoing, 1 own incoming, 2.. the colleague
// in direction dir (dir != 13, dx fastest)
__device__ inline int slot_of_dir(int dir) { return 2 + (dir < 13 ? dir : dir - 1); }
__device__ inline int dir_of_slot(int s) { return (s - 2) + ((s - 2) >= 13 ? 1 : 0); }

// Receivers of an accepted move (update_shift, src/tree.cpp:484-579): per
// path level own out, own inc and non-leaf colleagues' inc. A vector that
// both paths touch becomes one receiver carrying both contributions, so the
// update needs a single launch without write races. Receivers are matched by
// box coordinates (known from the header), the records go to T.recv and the
// count is returned to every thread. Block-cooperative.
__device__ int build_receivers(const DevTree& T, const Header& h, Receiver* out) {
  constexpr int PER = 28 * MAXLV;
  __shared__ int ckey[2 * PER];  // receiving node (-1 none)
  __shared__ signed char cfl[2 * PER][3];
  __shared__ short cmatch[2 * PER];
  __shared__ int wsum[32];
  const int levels = max(T.pw_hi - 1, 0);
  const int per = 28 * levels;
  const int ncand = 2 * per;
  const int ut = min(h.depth_t - 1, T.pw_hi), uo = min(h.depth_o - 1, T.pw_hi);
  for (int c = threadIdx.x; c < ncand; c += blockDim.x) {
    const int p = c / per, r = c % per;
    const int l = 2 + r / 28, s = r % 28;
    int recv = -1;
    signed char f[3] = {0, 0, 0};
    if (l <= (p == 0 ? ut : uo)) {
      const int node = p == 0 ? h.path_t[l] : h.path_o[l];
      recv = node;
      if (s >= 2) {
        const int dir = dir_of_slot(s);
        recv = T.col27[size_t(node) * 27 + dir];
        if (recv >= 0 && T.node_child0[recv] < 0) recv = -1;
        if (recv >= 0) {
          // source-centric image flag: periodic_shift(c_source, c_receiver)
          const int* X = p == 0 ? h.Xt[l] : h.Xo[l];
          const int dv[3] = {dir % 3 - 1, (dir / 3) % 3 - 1, dir / 9 - 1};
          for (int q = 0; q < 3; ++q) {
            const int v = X[q] + dv[q];
            f[q] = v < 0 ? 1 : (v >= (1 << l) ? -1 : 0);
          }
        }
      }
    }
    ckey[c] = recv;
    cfl[c][0] = f[0];
    cfl[c][1] = f[1];
    cfl[c][2] = f[2];
    cmatch[c] = -1;
  }
  __syncthreads();
  // an origin receiver equals a target receiver when it is the same vector;
  // its slot among the target's follows from the box coordinates
  for (int c = per + threadIdx.x; c < ncand; c += blockDim.x) {
    const int recv = ckey[c];
    if (recv < 0) continue;
    const int r = c - per, l = 2 + r / 28, s = r % 28;
    if (l > ut) continue;
    const int e = 1 << l;
    int ts;
    if (s == 0) {
      ts = h.path_t[l] == recv ? 0 : -1;
    } else {
      // receiver coordinates relative to the target's box at this level
      const int dir_o = s == 1 ? 13 : dir_of_slot(s);
      const int dvo[3] = {dir_o % 3 - 1, (dir_o / 3) % 3 - 1, dir_o / 9 - 1};
      int dir = 0, mul = 1;
      bool ok = true;
      for (int q = 0; q < 3; ++q) {
        int dq = ((h.Xo[l][q] + dvo[q] + e) & (e - 1)) - h.Xt[l][q];
        if (dq == e - 1) dq = -1;
        if (dq == 1 - e) dq = 1;
        ok = ok && dq >= -1 && dq <= 1;
        dir += (dq + 1) * mul;
        mul *= 3;
      }
      ts = !ok ? -1 : (dir == 13 ? 1 : slot_of_dir(dir));
    }
    if (ts >= 0) {
      const int t = (l - 2) * 28 + ts;
      if (ckey[t] == recv) {
        cmatch[c] = short(t);
        cmatch[t] = short(c);
      }
    }
  }
  __syncthreads();
  // compact: target receivers in slot order, then unmatched origin receivers
  const int per_thread = (ncand + blockDim.x - 1) / blockDim.x;
  const int c0 = threadIdx.x * per_thread;
  int cnt = 0;
  for (int c = c0; c < min(c0 + per_thread, ncand); ++c) cnt += ckey[c] >= 0 && (c < per || cmatch[c] < 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) {
      int v = wsum[w];
      wsum[w] = s;
      s += v;
    }
    wsum[31] = s;
  }
  __syncthreads();
  int pos = wsum[warp] + x - cnt;
  const int base = T.pw_base;
  for (int c = c0; c < min(c0 + per_thread, ncand); ++c) {
    if (!(ckey[c] >= 0 && (c < per || cmatch[c] < 0))) continue;
    const int r = c % per;
    Receiver R;
    R.off = ckey[c] - base;
    R.is_out = (r % 28) == 0;
    R.level = static_cast<signed char>(2 + r / 28);
    const bool is_t = c < per;
    const int m = cmatch[c];
    R.has_t = is_t;
    R.has_o = !is_t || m >= 0;
    for (int q = 0; q < 3; ++q) {
      R.ft[q] = is_t ? cfl[c][q] : 0;
      R.fo[q] = is_t ? (m >= 0 ? cfl[m][q] : 0) : cfl[c][q];
    }
    R.pad[0] = R.pad[1] = 0;
    out[pos++] = R;
  }
  const int total = wsum[31];
  __syncthreads();
  return total;
}

// ---------------------------------------------------------------------------
// Deferred expansion updates of a Metropolis sequence. An accepted move would
// read and write about 40 expansion rows (own outgoing and incoming rows and
// the colleagues' incoming rows of every path level: 39 MB at N = 1e5, 9
// digits, 10 us from L2). A long sequence keeps its accepted moves in a list
// instead and leaves the rows as they were at its start; the incoming row of a
// box B of level l then lacks, for each listed point a (weight w_a = +q at the
// target, -q at the origin) whose level-l box is B or one of its colleagues,
//   w_a conj(exp(-i k.(x_a - s_a L)))       (s_a: the image of a next to B),
// and the difference sum of a candidate point x of charge q in B lacks
//   c_l q w_a sum_k D(k) cos(k.d),  d = x - x_a + s_a L.
// D depends on |k| only, so the sum over the stored half grid folds onto the
// octant m = |k| / dk >= 0 per axis:
//   sum_{mz,my,mx >= 0} Dw[mz][my][mx] cos(mz tz) cos(my ty) cos(mx tx),  t = dk_l d,
// with Dw the table times the number of (kx, ky) signs: (n + 1)^3 multiply-adds
// for a pair of points, where an update row takes (n + 1) (2 n + 1)^2 complex
// read-modify-writes. When the sequence ends the rows are brought up to date
// once for all its moves (k_flush_outgoing, then the incoming pass).
template <int NP>
struct ModesOf {  // modes per half axis of the digits setting whose residual polynomial has NP terms
  static constexpr int ND = NP == 7 ? 6 : NP == 13 ? 12 : NP == 19 ? 19 : 26;
  static constexpr int NW = NP == 7 ? 4 : NP == 13 ? 8 : NP == 19 ? 13 : 17;
  static constexpr int ROWS = (ND + 1) * (ND + 1);  // (mz, my) rows of the folded table
  static constexpr int MT = (ROWS + 7) / 8;         // row tiles of the FP64 tensor product
  static constexpr int KS = (ND + 1 + 3) / 4;       // its steps of four mx
  // doubles from one mx to the next: a multiple of 8 rows, 4 modulo 16, so that
  // the eight rows and four mx of an operand load fall on different banks
  static constexpr int STR = 8 * MT + (20 - 8 * MT % 16) % 16;
  static constexpr int OCT = 4 * KS * STR;          // the folded table, zero past its rows and modes
  static constexpr int CT = 3 * 4 * KS * 4;         // cosines of one unit
};

}  // namespace

// an accepted move: point 0 its target (+), point 1 its origin (-); X the box
// coordinates at level u, the deepest expansion level on the point's path
struct Pending {
  double x[2][3];
  double q;
  int X[2][3];
  int u[2];
};

namespace {

__device__ inline void fill_pending(const DevTree& T, const Header& h, Pending& e) {
  const int ut = min(h.depth_t - 1, T.pw_hi), uo = min(h.depth_o - 1, T.pw_hi);
  e.q = h.q;
  e.u[0] = ut;
  e.u[1] = uo;
  for (int a = 0; a < 3; ++a) {
    e.x[0][a] = h.xt[a];
    e.x[1][a] = h.xo[a];
    e.X[0][a] = ut >= 0 ? h.Xt[ut][a] : 0;
    e.X[1][a] = uo >= 0 ? h.Xo[uo][a] : 0;
  }
}

// the box offset c - a of two box coordinates at a level of `side` boxes, and
// the image s in {-1, 0, 1} the offset was wrapped by; |offset| > 1: no neighbours
__device__ inline int box_offset(int c, int a, int side, int& s) {
  const int d = c - a;
  s = d == side - 1 ? 1 : (d == 1 - side ? -1 : 0);
  return d - s * side;
}

// the folded difference table: element (mx, my, mz) at mx STR + mz (n + 1) + my
__global__ void k_fold_d2(DevTree T, int stride, int total, double* out) {
  const int n = T.n_diff, n1 = n + 1, d = 2 * n + 1;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int mx = i / stride, r = i % stride, mz = r / n1, my = r % n1;
  double v = 0.0;
  if (mx < n1 && mz < n1) v = T.D2[((n - mz) * d + n + my) * d + n + mx] * (mx ? 2.0 : 1.0) * (my ? 2.0 : 1.0);  // kz < 0 entries carry the factor 2
  out[i] = v;
}

// is a listed move's target or origin a neighbour (or the box itself) of the
// candidate's target (pc = 0) or origin (pc = 1) box at level l?
__device__ inline bool pair_near(const Header& h, const Pending& e, int l, int pc, int pp) {
  const int top = (pc == 0 ? h.depth_t : h.depth_o) - 2;
  if (l > top || l > e.u[pp]) return false;
  const int* Xc = pc == 0 ? h.Xt[l] : h.Xo[l];
  bool ok = true;
  for (int a = 0; a < 3; ++a) {
    int s;
    ok = ok && abs(box_offset(Xc[a], e.X[pp][a] >> (e.u[pp] - l), 1 << l, s)) <= 1;
  }
  return ok;
}

// Which (listed move, level) units interact with the candidate, compacted in
// order by the calling warp into act[] as 256 entry + 16 flags + level (flags:
// bit 2 pc + pp for a pair of neighbouring points), the number returned to all
// its lanes.
__device__ __noinline__ int near_units(const Header& h, const Pending* list, int n_list, int* act) {
  const int lane = threadIdx.x & 31;
  const int top = max(h.depth_t, h.depth_o) - 2, nlev = top - 1;  // levels 2 .. top
  int n = 0;
  if (nlev > 0)
    for (int b = 0; b < n_list * nlev; b += 32) {
      const int i = b + lane;
      int flags = 0;
      const int en = i / nlev, l = 2 + i % nlev;
      if (i < n_list * nlev) {
        const Pending& e = list[en];
#pragma unroll
        for (int p = 0; p < 4; ++p) flags |= int(pair_near(h, e, l, p >> 1, p & 1)) << p;
      }
      const unsigned m = __ballot_sync(0xffffffffu, flags != 0);
      if (flags) act[n + __popc(m & ((1u << lane) - 1u))] = 256 * en + 16 * flags + l;
      n += __popc(m);
    }
  return n;
}

// Cosines of one unit by one warp, ct[axis][m][pair] = cos(m t): pair 2 pc + pp
// is the candidate's target (pc = 0) or origin against the listed move's target
// (pp = 0) or origin; the z axis carries the pair's sign, zero for a pair that
// does not interact. Lanes 0..23 take (pair, axis, parity of m): exp(i t), then
// steps of exp(2 i t).
template <int ND>
__device__ __noinline__ void unit_cosines(double L, double dk, const Header& h, const Pending& e, int unit, double* ct) {
  constexpr int N1 = ND + 1, KP = 4 * ((N1 + 3) / 4);
  const int lane = threadIdx.x & 31, l = unit & 15;
  if (lane < 4 * (KP - N1)) ct[N1 * 4 + lane] = 0.0;  // the x axis past its last mode
  if (lane < 24) {
    const int pair = lane / 6, axis = (lane >> 1) % 3, odd = lane & 1;
    const int pc = pair >> 1, pp = pair & 1;
    const bool near = (unit >> (4 + pair)) & 1;
    double sgn = 1.0, th = 0.0;
    if (axis == 2) sgn = near ? (pc == pp ? 1.0 : -1.0) : 0.0;
    if (near) {
      const int* Xc = pc == 0 ? h.Xt[l] : h.Xo[l];
      int s;
      box_offset(Xc[axis], e.X[pp][axis] >> (e.u[pp] - l), 1 << l, s);
      th = dk * ((pc == 0 ? h.xt[axis] : h.xo[axis]) - e.x[pp][axis] - s * L);
    }
    double sn, cs;
    sincos(th, &sn, &cs);
    const double2 z1 = make_double2(cs, sn), st = cmul(z1, z1);
    double2 v = odd ? make_double2(cs * sgn, sn * sgn) : make_double2(sgn, 0.0);
    double* dst = ct + axis * KP * 4 + pair;
    for (int m = odd; m < N1; m += 2) {
      dst[m * 4] = v.x;
      v = cmul(v, st);
    }
  }
}

// This lane's part of the pair sums of two units (their cosines side by side at
// ct; `two` false: the second is absent), the units' factors w0 and w1 applied.
// The inner sum over mx is a product of the folded table (rows (mz, my)) with
// eight columns of cosines, done on the FP64 tensor pipe (mma m8n8k4): the FMA
// pipe runs at the same rate, but there each table value and each cosine had
// to reach every lane's registers (4 wavefronts for a 16-byte broadcast), and
// shared memory held a unit at 2 290 cycles of an SM; its floor is 500. The
// calling warp takes row tiles t0, t0 + step, ...
template <int ND>
__device__ __forceinline__ double unit_pair_rows(const double* __restrict__ oct, const double* __restrict__ ct, bool two,
                                                 double w0, double w1, int t0, int step) {
  using MO = ModesOf<ND == 6 ? 7 : ND == 12 ? 13 : ND == 19 ? 19 : 25>;
  constexpr int N1 = ND + 1, KP = 4 * MO::KS;
  const int lane = threadIdx.x & 31, q4 = lane & 3, q8 = lane >> 2;
  double b[MO::KS];
#pragma unroll
  for (int k = 0; k < MO::KS; ++k) b[k] = (q8 < 4 || two) ? ct[(q8 >> 2) * MO::CT + (4 * k + q4) * 4 + (q8 & 3)] : 0.0;
  const int u = q4 >> 1;  // the unit of this lane's two result columns
  const double* cy = ct + u * MO::CT + KP * 4 + 2 * (q4 & 1);
  const double* cz = cy + KP * 4;
  const bool act = u == 0 || two;
  double out = 0.0;
#pragma unroll 2
  for (int t = t0; t < MO::MT; t += step) {
    const double* ap = oct + q4 * MO::STR + 8 * t + q8;
    double c0 = 0.0, c1 = 0.0;
#pragma unroll
    for (int k = 0; k < MO::KS; ++k)
      asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
          : "+d"(c0), "+d"(c1)
          : "d"(ap[4 * k * MO::STR]), "d"(b[k]));
    const int r = 8 * t + q8;
    if (act && r < MO::ROWS) {
      const int mz = r / N1, my = r % N1;
      const double2 y = *reinterpret_cast<const double2*>(cy + my * 4), z = *reinterpret_cast<const double2*>(cz + mz * 4);
      out = fma(c0 * y.x, z.x, out);
      out = fma(c1 * y.y, z.y, out);
    }
  }
  return out * (u ? w1 : w0);
}

// This thread's part of the difference sums of both paths (energy_shift.cpp:
// 92-140), modes threadIdx.x, threadIdx.x + T, ... of every level. What bounds it
// is the rows' way from L2: a box that both paths share is read once (most
// trial moves stay in their box), and ILP modes are loaded before the first is
// used.
template <int ND, int T, int ILP>
__device__ double diff_sum(const DevTree& tr, const Header& h, const Tables& oo, const Tables& to, int lo_max, int lt_max,
                           const double* c_level) {
  constexpr int D = 2 * ND + 1, H = (ND + 1) * D * D;
  double e = 0;
  for (int l = 2; l <= max(lo_max, lt_max); ++l) {
    const bool has_o = l <= lo_max, has_t = l <= lt_max;
    const bool same = has_o && has_t && h.path_o[l] == h.path_t[l];
    const double2* ro = has_o ? tr.inc + size_t(h.path_o[l] - tr.pw_base) * H : nullptr;
    const double2* rt = has_t && !same ? tr.inc + size_t(h.path_t[l] - tr.pw_base) * H : nullptr;
    double s = 0;
    for (int k0 = threadIdx.x; k0 < H; k0 += T * ILP) {
      double2 co[ILP], cn[ILP];
      double dv[ILP];
#pragma unroll
      for (int j = 0; j < ILP; ++j) {
        const int k = k0 + j * T;
        dv[j] = k < H ? tr.D2[k] : 0.0;
        if (k < H && ro) co[j] = ro[k];
        if (k < H && rt) cn[j] = rt[k];
      }
#pragma unroll
      for (int j = 0; j < ILP; ++j) {
        const int k = k0 + j * T;
        if (k >= H) break;
        const int ix = k % D, iy = (k / D) % D, iz = k / (D * D);
        double v = 0;
        if (has_o) {
          const double2 o = cmul(oo.lev[l][2][iz], cmul(oo.lev[l][1][iy], oo.lev[l][0][ix]));
          v -= o.x * co[j].x - o.y * co[j].y - (o.x * o.x + o.y * o.y);
        }
        if (has_t) {
          const double2 c = same ? co[j] : cn[j];
          const double2 t = cmul(to.lev[l][2][iz], cmul(to.lev[l][1][iy], to.lev[l][0][ix]));
          v += t.x * c.x - t.y * c.y;
        }
        s += v * dv[j];
      }
    }
    e += s * c_level[l];
  }
  return e;
}

// Outgoing rows at the end of a sequence: out_B += sum of the listed points
// whose path passes through B. Blocks (node, part of the row); a node no move
// touched returns at once. Points are taken 8 at a time in list order: their
// phase tables go to shared memory (one sincos per entry, as build_tables),
// then each thread adds them to its modes. FP64-bound: 10 operations per point
// and mode.
constexpr int FO_T = 256, FO_PTS = 8, FO_PARTS = 8;

template <int ND>
__device__ __forceinline__ void flush_row(const DevTree& T, const Pending* __restrict__ list,
                                          const int* __restrict__ n_list, const int* __restrict__ touched) {
  constexpr int D = 2 * ND + 1, H = (ND + 1) * D * D, TAB = 3 * D;
  __shared__ double2 tab[FO_PTS][TAB];
  __shared__ int sel[FO_PTS];
  __shared__ int s_n, s_next;
  // level-2 nodes in FO_PARTS parts, the others whole
  const int n2 = T.level_start[3] - T.level_start[2];
  int node = T.pw_base, part = 0, parts = 1;
  if (int(blockIdx.x) < n2 * FO_PARTS) {
    node += blockIdx.x / FO_PARTS;
    part = blockIdx.x % FO_PARTS;
    parts = FO_PARTS;
  } else {
    node += n2 + int(blockIdx.x) - n2 * FO_PARTS;
  }
  if (touched[node - T.pw_base] == 0) return;
  const int l = T.node_level[node];
  const uint64_t pf = T.node_prefix[node];
  const int X[3] = {int(compact3(pf)), int(compact3(pf >> 1)), int(compact3(pf >> 2))};
  const int n = *n_list;
  const int k0 = int(long(H) * part / parts), k1 = int(long(H) * (part + 1) / parts);
  double2* row = T.out + size_t(node - T.pw_base) * H;
  if (threadIdx.x == 0 && part == 0) atomicAdd(&T.work[1], 32ull * H);
  int at = 0;  // points are 2 n: (move, target / origin)
  while (at < 2 * n) {
    // warp 0 collects the next points of this node, in list order
    if (threadIdx.x < 32) {
      int cnt = 0;
      int b = at;
      for (; b < 2 * n && cnt < FO_PTS; b += 32) {
        const int i = b + threadIdx.x;
        bool in = false;
        if (i < 2 * n) {
          const Pending& e = list[i >> 1];
          const int p = i & 1, u = e.u[p];
          in = u >= l && (e.X[p][0] >> (u - l)) == X[0] && (e.X[p][1] >> (u - l)) == X[1] &&
               (e.X[p][2] >> (u - l)) == X[2];
        }
        unsigned m = __ballot_sync(0xffffffffu, in);
        const int room = FO_PTS - cnt;
        const int rank = __popc(m & ((1u << threadIdx.x) - 1u));
        if (in && rank < room) sel[cnt + rank] = i;
        if (__popc(m) > room) {  // full: the scan goes on after the last point taken
          int last = 0;
          for (int k = 0; k < room; ++k) {
            last = __ffs(m) - 1;
            m &= m - 1;
          }
          cnt = FO_PTS;
          b = b + last + 1 - 32;
        } else {
          cnt += __popc(m);
        }
      }
      if (threadIdx.x == 0) {
        s_n = cnt;
        s_next = b;
      }
    }
    __syncthreads();
    const int cnt = s_n;
    at = s_next;
    for (int t = threadIdx.x; t < cnt * TAB; t += FO_T) {
      const int c = t / TAB, r = t % TAB, axis = r / D, m = r % D - ND;
      const Pending& e = list[sel[c] >> 1];
      const int p = sel[c] & 1;
      const double th = level_dk(T, l) * (e.x[p][axis] - center_of(T.L, l, X[axis]));
      double sn, cs;
      sincos(-double(m) * th, &sn, &cs);
      const double sc = axis == 2 ? (p == 0 ? e.q : -e.q) : 1.0;
      tab[c][r] = cmul(make_double2(cs * sc, sn * sc), root6(-(2 * X[axis] + 1) * m));
    }
    __syncthreads();
    if (cnt > 0)
      for (int k = k0 + threadIdx.x; k < k1; k += FO_T) {
        const int ix = k % D, iy = (k / D) % D, iz = k / (D * D);
        double2 v = row[k];
        for (int c = 0; c < cnt; ++c) v = cadd(v, cmul(tab[c][2 * D + iz], cmul(tab[c][D + iy], tab[c][ix])));
        row[k] = v;
      }
    __syncthreads();
  }
}

// blocks of a tree
inline int flush_blocks(const DevTree& D) {
  const int n_pw = D.pw_hi >= D.pw_lo ? D.level_start[D.pw_hi + 1] - D.pw_base : 0;
  return n_pw > 0 ? n_pw + (FO_PARTS - 1) * (D.level_start[3] - D.level_start[2]) : 0;
}

template <int ND>
__global__ void __launch_bounds__(FO_T) k_flush_outgoing(DevTree T, const Pending* __restrict__ list,
                                                         const int* __restrict__ n_list,
                                                         const int* __restrict__ touched) {
  flush_row<ND>(T, list, n_list, touched);
}

// the rows of a set of trees
template <int ND>
__global__ void __launch_bounds__(FO_T) k_flush_set(const DevTree* __restrict__ trees, const SequenceRows* __restrict__ rows,
                                                    int n) {
  const int t = set_tree();
  if (t >= n) return;
  const SequenceRows r = rows[t];
  const DevTree& T = trees[t];
  if (r.n_pw == 0 || *r.n_list == 0 || int(blockIdx.x) >= r.n_pw + (FO_PARTS - 1) * (T.level_start[3] - T.level_start[2]))
    return;
  flush_row<ND>(T, r.list, r.n_list, r.touched);
}

// empties the lists of a set of trees
__global__ void k_clear_set(const SequenceRows* __restrict__ rows, int n) {
  const int t = set_tree();
  if (t >= n) return;
  const SequenceRows r = rows[t];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= r.n_pw; i += gridDim.x * blockDim.x) r.touched[i] = 0;
}

// the error words of a set of trees
__global__ void k_errors_of_set(const DevTree* __restrict__ trees, int n, int* __restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) err[i] = *trees[i].err;
}

struct ShiftArgs {
  const int* idx;
  const double* disp;
  const double* u;
  double beta;
  int move;
  int mode;  // 0: evaluate only, 1: Metropolis
  double* dE_out;
  int* acc_out;
  double c_window;  // dk_0^3 / (2 pi)^3
  double* partials;
  unsigned int* counter;
  Proposal* prop;
  double2* ptab;          // phase tables published for k_update
  long ptab_per;          // complex entries per path
  const MoveCursor* cur;  // non-null: proposals come from the cursor (captured graphs)
  double* host_out;       // dE and its five parts for the host (mapped memory; may be null)
};

// a proposal passed with the launch (ShiftArgs::idx null)
struct OneMove {
  int i;
  double d[3];
};

// Grid: blocks [0, G-3) do the plane-wave sums; block G-3 the target
// residual, block G-2 the origin residual, block G-1 lists the receivers of an
// update (beside the sums: behind them it lengthened the launch by 2 us). The
// last block to finish reduces.
template <int NP>
__global__ void __launch_bounds__(SH_T) k_shift(DevTree T, ShiftArgs a, const __grid_constant__ OneMove one) {
  extern __shared__ double2 sm2[];
  __shared__ Header h;
  __shared__ double red[4][32];
  __shared__ double c_level[MAXLV + 2];  // dk_l^3 / (2 pi)^3 * dscale_l
  __shared__ bool is_last;
  const ResidualPoly<NP> poly(T);
  if (threadIdx.x >= 2 && threadIdx.x < MAXLV + 2) {
    const double dk = level_dk(T, threadIdx.x);
    c_level[threadIdx.x] = dk * dk * dk / (8.0 * 3.14159265358979323846 * 3.14159265358979323846 *
                                           3.14159265358979323846) * level_dscale(threadIdx.x);
  }
  if (a.cur) {
    const MoveCursor c = *a.cur;
    a.idx = c.idx;
    a.disp = c.disp;
    a.u = c.u;
    a.dE_out = c.dE;
    a.acc_out = c.acc;
    a.mode = c.mode;
    a.beta = c.beta;
    a.move += c.off;
  }
  const int move = a.move;
  resolve(T, a.idx ? a.idx[move] : one.i, a.idx ? a.disp + 3 * move : one.d, h);
  const int G = gridDim.x;
  const int Gpw = G - 3;
  double acc[4] = {0, 0, 0, 0};  // window, difference, residual target, residual origin
  if (blockIdx.x < Gpw) {
    // dE needs the non-leaf path levels 2 .. depth-2; an accept-and-update
    // needs 2 .. min(depth-1, pw_hi): build the superset
    const int lo_max = h.depth_o - 2, lt_max = h.depth_t - 2;
    const int uo = min(h.depth_o - 1, T.pw_hi), ut = min(h.depth_t - 1, T.pw_hi);
    const int per = 3 * (2 * T.n_window + 1) + max(max(uo, ut) - 1, 0) * 3 * (2 * T.n_diff + 1);
    Tables to, oo;
    alloc_tables(sm2, T, oo);
    alloc_tables(sm2 + per, T, to);
    build_tables(T, h.xo, h.q, h.Xo, uo, oo, threadIdx.x, blockDim.x);
    build_tables(T, h.xt, h.q, h.Xt, ut, to, threadIdx.x, blockDim.x);
    __syncthreads();
    if (blockIdx.x == 0) {
      // publish the tables for k_update
      for (int p = 0; p < 2; ++p) {
        Tables g;
        alloc_tables(a.ptab + size_t(p) * a.ptab_per, T, g);
        const Tables& s = p == 0 ? oo : to;
        const int up = p == 0 ? uo : ut;
        for (int ax = 0; ax < 3; ++ax)
          for (int e = threadIdx.x; e < T.dw; e += blockDim.x) g.root[ax][e] = s.root[ax][e];
        for (int l = 2; l <= up; ++l)
          for (int ax = 0; ax < 3; ++ax)
            for (int e = threadIdx.x; e < T.dd; e += blockDim.x) g.lev[l][ax][e] = s.lev[l][ax][e];
      }
    }
    const int stride = Gpw * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    // window (src/energy_shift.cpp:72-90)
    for (int k = t0; k < T.Hw; k += stride) {
      double2 t = phase_at(to.root, k, T.dw), o = phase_at(oo.root, k, T.dw);
      double2 g = T.out_root[k];
      double ar = t.x - o.x, ai = t.y - o.y, br = g.x - o.x, bi = g.y - o.y;
      acc[0] += (ar * br + ai * bi) * T.W[k];
    }
    // difference (src/energy_shift.cpp:92-140), all path levels per mode
    const int base = T.pw_base;
    const int d = T.dd;
    for (int k = t0; k < T.H; k += stride) {
      const int ix = k % d, iy = (k / d) % d, iz = k / (d * d);
      double s = 0;
      for (int l = 2; l <= lo_max; ++l) {
        double2 o = cmul(oo.lev[l][2][iz], cmul(oo.lev[l][1][iy], oo.lev[l][0][ix]));
        double2 c = T.inc[size_t(h.path_o[l] - base) * T.H + k];
        s -= (o.x * c.x - o.y * c.y - (o.x * o.x + o.y * o.y)) * c_level[l];
      }
      for (int l = 2; l <= lt_max; ++l) {
        double2 t = cmul(to.lev[l][2][iz], cmul(to.lev[l][1][iy], to.lev[l][0][ix]));
        double2 c = T.inc[size_t(h.path_t[l] - base) * T.H + k];
        s += (t.x * c.x - t.y * c.y) * c_level[l];
      }
      acc[1] += s * T.D2[k];
    }
  } else if (blockIdx.x == Gpw) {
    const int lt = h.depth_t - 1;
    acc[2] = residual_sum(T, poly, h.path_t[lt], lt, h.Xt[lt], h.xt) * h.q;
  } else if (blockIdx.x == Gpw + 1) {
    const int lo = h.depth_o - 1;
    acc[3] = residual_sum(T, poly, h.path_o[lo], lo, h.Xo[lo], h.xo) * h.q;
  } else {
    const int n = build_receivers(T, h, T.recv);
    if (threadIdx.x == 0) a.prop->n_recv = n;
  }
  block_sum4(acc, red);
  if (threadIdx.x == 0) {
    double* pp = a.partials + 4 * size_t(blockIdx.x);
    for (int c = 0; c < 4; ++c) pp[c] = acc[c];
    __threadfence();
    unsigned prev = atomicAdd(a.counter, 1u);
    is_last = (prev == unsigned(G - 1));
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // fixed-order reduction of the block partials (deterministic)
  double tot[4] = {0, 0, 0, 0};
  for (int b = threadIdx.x; b < G; b += blockDim.x)
    for (int c = 0; c < 4; ++c) tot[c] += __ldcg(a.partials + 4 * size_t(b) + c);
  block_sum4(tot, red);
  if (threadIdx.x == 0) {
    const double dEw = tot[0] * a.c_window;  // 2 * sum * dk0^3 / (2 (2 pi)^3)
    const double d = tot[1], rt = tot[2], ro = tot[3];
    double self = 0;
    if (h.dr != 0) self = poly(h.dr, level_box(T, 2)) * h.q * h.q;
    const double dE = dEw + d + rt - ro - self;
    Proposal* P = a.prop;
    P->i_orig = h.i_orig;
    P->slot = h.slot;
    P->q = h.q;
    for (int c = 0; c < 3; ++c) {
      P->xo[c] = h.xo[c];
      P->xt[c] = h.xt[c];
    }
    P->depth_o = h.depth_o;
    P->depth_t = h.depth_t;
    for (int l = 0; l < MAXLV; ++l) {
      P->path_o[l] = l < h.depth_o ? h.path_o[l] : -1;
      P->path_t[l] = l < h.depth_t ? h.path_t[l] : -1;
    }
    P->dE = dE;
    P->parts[0] = dEw;
    P->parts[1] = d;
    P->parts[2] = rt;
    P->parts[3] = ro;
    P->parts[4] = self;
    if (a.host_out) {
      a.host_out[0] = dE;
      for (int c = 0; c < 5; ++c) a.host_out[1 + c] = P->parts[c];
    }
    int accd = 0;
    if (a.mode == 1) {
      const double u = a.u[move];
      accd = u < exp(-a.beta * dE) ? 1 : 0;
      if (a.acc_out) a.acc_out[move] = accd;
    }
    if (a.dE_out) a.dE_out[move] = dE;
    P->accepted = accd;
    P->valid = 1;
    *a.counter = 0u;
  }
}

// ---------------------------------------------------------------------------
// update_shift (src/tree.cpp:447-597) in one launch. Each thread owns one
// mode k (grid x) and walks a range of receivers (grid y): out += t - o, or
// inc += conj(t s_t) - conj(o s_o) with the periodic image phases s; the
// y == 0 blocks also update the root expansion (out += t; out -= o) and
// block (0, 0) commits the particle membership.
constexpr int UPD_T = 128;
constexpr int UPD_UNROLL = 8;

__device__ bool commit_move(const DevTree& T, const Proposal& P);

__global__ void __launch_bounds__(UPD_T) k_update(DevTree T, const double2* __restrict__ ptab, long ptab_per,
                                                  bool force, int* host_err) {
  __shared__ Receiver rs[MAX_RECV];
  __shared__ int s_acc, s_nr;
  if (threadIdx.x == 0) {
    s_acc = force || T.prop->accepted;
    s_nr = T.prop->n_recv;
  }
  __syncthreads();
  if (!s_acc) return;
  const int nr = s_nr;
  const int r0 = int((long(blockIdx.y) * nr) / gridDim.y), r1 = int((long(blockIdx.y + 1) * nr) / gridDim.y);
  for (int r = r0 + threadIdx.x; r < r1; r += blockDim.x) rs[r - r0] = T.recv[r];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    atomicAdd(&T.work[0], 1ull);
    atomicAdd(&T.work[1], 32ull * ((unsigned long long)T.Hw + (unsigned long long)nr * T.H));
    if (force) T.prop->accepted = 1;
    commit_move(T, *T.prop);
    if (host_err) *host_err = ldm<true>(T.err);
  }
  __syncthreads();
  Tables tt, to;
  alloc_tables(const_cast<double2*>(ptab) + ptab_per, T, tt);
  alloc_tables(const_cast<double2*>(ptab), T, to);
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.y == 0 && k < T.Hw) {
    double2 t = phase_at(tt.root, k, T.dw), o = phase_at(to.root, k, T.dw);
    double2 g = T.out_root[k];
    g = cadd(g, t);
    g = csub(g, o);
    T.out_root[k] = g;
  }
  if (k >= T.H) return;
  const int n = T.n_diff, d = T.dd;
  const int ix = k % d, iy = (k / d) % d, iz = k / (d * d);
  const int a0 = ((ix - n) % 3 + 3) % 3, a1 = ((iy - n) % 3 + 3) % 3, a2 = ((iz - n) % 3 + 3) % 3;
  int r = 0;
  const int nloc = r1 - r0;
  while (r < nloc) {
    // a run of receivers on one level shares the two single-particle phases
    const int l = rs[r].level;
    int re = r + 1;
    while (re < nloc && rs[re].level == l) ++re;
    const double2 pt0 = cmul(tt.lev[l][2][iz], cmul(tt.lev[l][1][iy], tt.lev[l][0][ix]));
    const double2 po0 = cmul(to.lev[l][2][iz], cmul(to.lev[l][1][iy], to.lev[l][0][ix]));
    const double2 pt1 = cmul(pt0, root6(-2)), pt2 = cmul(pt0, root6(-4));
    const double2 po1 = cmul(po0, root6(-2)), po2 = cmul(po0, root6(-4));
    const int two_l = (l & 1) ? 2 : 1;
    for (; r < re; r += UPD_UNROLL) {
      double2 v[UPD_UNROLL];
      size_t off[UPD_UNROLL];
#pragma unroll
      for (int u = 0; u < UPD_UNROLL; ++u) {
        if (r + u < re) {
          const Receiver& R = rs[r + u];
          off[u] = size_t(R.off) * T.H + k;
          v[u] = R.is_out ? T.out[off[u]] : T.inc[off[u]];
        }
      }
#pragma unroll
      for (int u = 0; u < UPD_UNROLL; ++u) {
        if (r + u < re) {
          const Receiver& R = rs[r + u];
          // image phase: a cube root of unity, w^-e with e in [-12, 12] mod 3
          const int et = ((a0 * R.ft[0] + a1 * R.ft[1] + a2 * R.ft[2]) * two_l + 12) % 3;
          const int eo = ((a0 * R.fo[0] + a1 * R.fo[1] + a2 * R.fo[2]) * two_l + 12) % 3;
          double2 del = make_double2(0.0, 0.0);
          if (R.has_t) del = et == 0 ? pt0 : (et == 1 ? pt1 : pt2);
          if (R.has_o) del = csub(del, eo == 0 ? po0 : (eo == 1 ? po1 : po2));
          if (R.is_out) T.out[off[u]] = cadd(v[u], del);
          else T.inc[off[u]] = make_double2(v[u].x + del.x, v[u].y - del.y);
        }
      }
    }
    r = re;
  }
}

// particle membership and position (exact on every level); one thread. The
// independent loads are issued together and the per-level counts change by
// atomic adds that need no reply, so the thread waits on few round trips.
//
// False when the particle stays where it is: its arrival finds both the target
// leaf and the overflow pool full, or (after such a move, by which the caller's
// idea of its place may be wrong) its slot is not one of the leaf it is said to
// leave. The error word then says so; slots, pool and counts stay as they were, so
// whatever runs before the host reads it finds every particle in one place.
__device__ bool commit_move(const DevTree& T, const Proposal& P) {
  if (!P.accepted) return true;
  const int leafA = P.path_o[P.depth_o - 1];
  const int leafB = P.path_t[P.depth_t - 1];
  const int i = P.i_orig;
  const int s = P.slot;
  const double xt0 = P.xt[0], xt1 = P.xt[1], xt2 = P.xt[2], q = P.q;
  const bool pooled = s >= T.n_slots;
  const int cA = T.leaf_count[leafA], begA = T.node_begin[leafA];
  const int cB = T.leaf_count[leafB], begB = T.node_begin[leafB], endB = T.node_end[leafB];
  const int pn = *T.pool_n;
  const bool there = pooled ? T.p_leaf[s - T.n_slots] == leafA && T.p_orig[s - T.n_slots] == i : s >= begA && s < begA + cA;
  if (!there || (leafA != leafB && begB + cB >= endB && pn >= T.pool_cap)) {
    atomicOr(T.err, 1);
    return false;
  }
  if (leafA == leafB) {
    if (!pooled) {
      T.sx[s] = xt0;
      T.sy[s] = xt1;
      T.sz[s] = xt2;
    } else {
      const int p = s - T.n_slots;
      T.px[p] = xt0;
      T.py[p] = xt1;
      T.pz[p] = xt2;
    }
    return true;
  }
  // remove from the origin leaf (swap with its last particle) or the pool
  if (!pooled) {
    const int last = begA + cA - 1;
    const int ol = T.s_orig[last];
    const double lx = T.sx[last], ly = T.sy[last], lz = T.sz[last], lq = T.sq[last];
    const uint64_t pfx = T.node_prefix[leafA];
    const int lvl = T.node_level[leafA];
    if (s != last) {
      T.sx[s] = lx;
      T.sy[s] = ly;
      T.sz[s] = lz;
      T.sq[s] = lq;
      T.s_orig[s] = ol;
      T.orig_slot[ol] = s;
    }
    // a freed slot holds a zero charge at its leaf's centre
    T.sx[last] = center_of(T.L, lvl, int(compact3(pfx)));
    T.sy[last] = center_of(T.L, lvl, int(compact3(pfx >> 1)));
    T.sz[last] = center_of(T.L, lvl, int(compact3(pfx >> 2)));
    T.sq[last] = 0.0;
    T.s_orig[last] = -1;
    T.leaf_count[leafA] = cA - 1;
  } else {
    const int p = s - T.n_slots;
    T.p_orig[p] = -1;
    T.pq[p] = 0.0;
  }
  // insert into the target leaf, or park in the pool when it is full
  const int slot = begB + cB;
  if (slot < endB) {
    T.sx[slot] = xt0;
    T.sy[slot] = xt1;
    T.sz[slot] = xt2;
    T.sq[slot] = q;
    T.s_orig[slot] = i;
    T.orig_slot[i] = slot;
    T.leaf_count[leafB] = cB + 1;
  } else {
    T.px[pn] = xt0;
    T.py[pn] = xt1;
    T.pz[pn] = xt2;
    T.pq[pn] = q;
    T.p_orig[pn] = i;
    T.p_leaf[pn] = leafB;
    T.orig_slot[i] = T.n_slots + pn;
    *T.pool_n = pn + 1;
  }
  for (int l = 0; l < P.depth_o; ++l) atomicAdd(T.node_count + P.path_o[l], -1);
  for (int l = 0; l < P.depth_t; ++l) atomicAdd(T.node_count + P.path_t[l], 1);
  return true;
}


// ---------------------------------------------------------------------------
// Persistent Metropolis kernel: one cooperative launch runs a whole sequence
// of trial moves on every SM. Per move, every block resolves the proposal and
// builds both paths' phase tables itself (no broadcast needed), adds its share
// of the window, difference and near-field sums, and publishes 4 partials;
// after a grid barrier every block reduces all partials in the same fixed
// order, so all blocks reach the same dE and the same Metropolis decision. An
// accepted move is then applied by all blocks (receivers listed per block,
// one read-modify-write per mode and vector), block 0 commits the particle,
// and a second barrier orders the update before the next move. Barrier waits
// are bounded; a wait that gives up sets an error bit and every block returns.
constexpr int MC_T = 512;

struct McArgs {
  const int* idx;
  const double* disp;
  const double* u;
  double beta;
  int n_moves;
  double* dE_out;
  int* acc_out;
  double c_window;          // dk_0^3 / (2 pi)^3
  double* partials;         // [2][G][4], double-buffered by move parity
  unsigned int* arrivals;   // barrier arrivals, zero at launch
  long long spin_limit;     // polls before a barrier wait gives up
};

__device__ inline unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier over a monotonically increasing arrival counter, as an
// arrival and a wait that may be apart; nbar counts the barriers this block
// has arrived at (kept by thread 0).
__device__ void mc_arrive(const McArgs& a, unsigned& nbar) {
  __syncthreads();
  if (threadIdx.x == 0) {
    ++nbar;
    // the release orders this block's writes (made visible to this thread by
    // the __syncthreads above) before the arrival; no reply is awaited
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.arrivals) : "memory");
  }
}

// Waits until every block has arrived at this block's last barrier. False
// when the wait gave up or another block reported a failure.
__device__ bool mc_wait(const DevTree& T, const McArgs& a, unsigned nbar) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    const unsigned target = nbar * gridDim.x;
    int ok = 1;
    for (long long it = 0;; ++it) {
      if (ld_acquire(a.arrivals) >= target) break;
      if (ldm<true>(T.err) & 2) {
        ok = 0;
        break;
      }
      if (it >= a.spin_limit) {
        atomicOr(T.err, 2);
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
    // the acquire load above orders this thread after the other blocks'
    // releases; the barrier below passes that order on to the whole block
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ bool mc_barrier(const DevTree& T, const McArgs& a, unsigned& nbar) {
  mc_arrive(a, nbar);
  return mc_wait(T, a, nbar);
}

// Source lists of one path's leaf for the near field: the leaf, its 26
// colleagues and 8 coarse neighbours, with their periodic offsets.
struct ResMeta {
  int beg[36], cnt[36], pre[37], lvl[36];
  unsigned long long pfx[36];
  double off[36][3];
};

__device__ void res_meta(const DevTree& T, int leaf, int l, const int* Xl, int src, ResMeta& M) {
  const double b = level_box(T, l);
  int j = -1;
  if (src == 0) j = leaf;
  else if (src <= 27) j = (src - 1 == 13) ? -1 : T.col27[size_t(leaf) * 27 + (src - 1)];
  else j = T.coarse8[size_t(leaf) * 8 + (src - 28)];
  int beg = 0, cnt = 0, lj = 0;
  unsigned long long pj = 0;
  double off[3] = {0, 0, 0};
  if (j >= 0) {
    lj = T.node_level[j];
    pj = T.node_prefix[j];
    const int ch = T.node_child0[j];
    beg = T.node_begin[j];
    const int end = ch < 0 ? beg + ldm<true>(T.leaf_count + j) : T.node_end[j];
    cnt = end - beg;
    const double bj = level_box(T, lj);
    const int Xj[3] = {int(compact3(pj)), int(compact3(pj >> 1)), int(compact3(pj >> 2))};
    for (int d = 0; d < 3; ++d)
      off[d] = -periodic_shift_d(center_of(T.L, l, Xl[d]), center_of(T.L, lj, Xj[d]), T.L, b, bj) * T.L;
  }
  M.beg[src] = beg;
  M.cnt[src] = j >= 0 ? cnt : -1;
  M.lvl[src] = lj;
  M.pfx[src] = pj;
  for (int d = 0; d < 3; ++d) M.off[src][d] = off[d];
}

template <int NP>
__global__ void __launch_bounds__(MC_T, 1) k_mc(DevTree T, McArgs a) {
  extern __shared__ double2 sm2[];
  __shared__ Header h;
  __shared__ double red[4][32];
  __shared__ double c_level[MAXLV + 2];
  __shared__ ResMeta meta[2];
  __shared__ Receiver rs[MAX_RECV];
  __shared__ Proposal P;
  __shared__ int s_acc;
  __shared__ int s_rounds[9];  // grid-stride rounds of H*g update units
  __shared__ int s_pn;         // overflow pool fill
  __shared__ int s_stale;      // the accepted move invalidated the preloaded next particle
  const ResidualPoly<NP> poly(T);
  if (threadIdx.x >= 1 && threadIdx.x <= 8) {
    const long units = long(T.H) * threadIdx.x, gs = long(gridDim.x) * blockDim.x;
    s_rounds[threadIdx.x] = int((units + gs - 1) / gs);
  }
  if (threadIdx.x >= 2 && threadIdx.x < MAXLV + 2) {
    const double dk = level_dk(T, threadIdx.x);
    c_level[threadIdx.x] = dk * dk * dk / (8.0 * 3.14159265358979323846 * 3.14159265358979323846 *
                                           3.14159265358979323846) * level_dscale(threadIdx.x);
  }
  const int G = gridDim.x;
  const int gt = blockIdx.x * blockDim.x + threadIdx.x, gstride = G * blockDim.x;
  // window and root items run from the end of the grid, the difference and
  // update units from its start, so no block carries both
  const int gtr = gstride - 1 - gt;
  unsigned nbar = 0;
  // warp 0 runs one proposal ahead: the next index and displacement are
  // loaded at the top of a move, the next slot after the sums and the
  // particle itself after the decision, so the next resolve starts from them
  // unless the accepted move changed that slot or particle
  int i_cur = threadIdx.x < 32 ? a.idx[0] : 0;
  double d_cur[3] = {0, 0, 0};
  if (threadIdx.x < 32)
    for (int c = 0; c < 3; ++c) d_cur[c] = a.disp[c];
  Preload pre{-1, 0, 0, 0, 0};
  // An accepted move ends with an arrival at a grid barrier whose wait is
  // deferred: the next move's resolve and phase tables read only the
  // preloaded particle and the static refinement bitmaps, so they run before
  // the wait; the near-field source lists, the pool fill and the sums, which
  // read what other blocks update or commit, run after it. When the accepted
  // move invalidated the preload, the wait comes first.
  bool pend = false;
  for (int m = 0; m < a.n_moves; ++m) {
    const bool more = threadIdx.x < 32 && m + 1 < a.n_moves;
    const int i_next = more ? a.idx[m + 1] : 0;
    double d_next[3] = {0, 0, 0};
    if (more)
      for (int c = 0; c < 3; ++c) d_next[c] = a.disp[3 * (m + 1) + c];
    if (pend && s_stale) {
      if (!mc_wait(T, a, nbar)) return;
      pend = false;
    }
    resolve<true>(T, i_cur, d_cur, h, &pre);
    const int lo_max = h.depth_o - 2, lt_max = h.depth_t - 2;
    // the incoming rows of both paths go to L2 while the tables are built
    for (int k = gt; k < T.H; k += gstride) {
      for (int l = 2; l <= lo_max; ++l)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(T.inc + size_t(h.path_o[l] - T.pw_base) * T.H + k));
      for (int l = 2; l <= lt_max; ++l)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(T.inc + size_t(h.path_t[l] - T.pw_base) * T.H + k));
    }
    const int uo = min(h.depth_o - 1, T.pw_hi), ut = min(h.depth_t - 1, T.pw_hi);
    const int per = 3 * (2 * T.n_window + 1) + max(max(uo, ut) - 1, 0) * 3 * (2 * T.n_diff + 1);
    Tables to, oo;
    alloc_tables(sm2, T, oo);
    alloc_tables(sm2 + per, T, to);
    // near-field source lists on threads 0..71, phase tables on the rest
    auto source_lists = [&]() {
      if (threadIdx.x == 0) s_pn = __ldcg(T.pool_n);
      const int p = threadIdx.x / 36, src = threadIdx.x % 36;
      const int lv = (p == 0 ? h.depth_t : h.depth_o) - 1;
      res_meta(T, p == 0 ? h.path_t[lv] : h.path_o[lv], lv, p == 0 ? h.Xt[lv] : h.Xo[lv], src, meta[p]);
    };
    if (threadIdx.x < 72) {
      if (!pend) source_lists();
    } else {
      const int nthr = blockDim.x - 72, t = threadIdx.x - 72;
      build_tables(T, h.xo, h.q, h.Xo, uo, oo, t, nthr);
      build_tables(T, h.xt, h.q, h.Xt, ut, to, t, nthr);
    }
    if (pend) {
      if (!mc_wait(T, a, nbar)) return;
      pend = false;
      if (threadIdx.x < 72) source_lists();
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      ResMeta& M = meta[threadIdx.x];
      int s = 0;
      for (int src = 0; src < 36; ++src) {
        M.pre[src] = s;
        s += max(M.cnt[src], 0);
      }
      M.pre[36] = s;
    }
    __syncthreads();
    double acc[4] = {0, 0, 0, 0};
    // near field of the target and the origin (src/energy_shift.cpp:233-302):
    // the pairs of both paths split evenly over the blocks. The first pair's
    // source is loaded before the mode sums so the two latencies overlap.
    const int nt = meta[0].pre[36], no = meta[1].pre[36], np = nt + no;
    const int e0 = int((long(blockIdx.x) * np) / G), e1 = int((long(blockIdx.x + 1) * np) / G);
    const double eps = 2.220446049250313e-16;
    int e = e0 + threadIdx.x;
    double4 src_first = make_double4(0, 0, 0, 0);
    int p_first = 0, srci_first = 0;
    if (e < e1) {
      p_first = e < nt ? 0 : 1;
      const ResMeta& M = meta[p_first];
      const int ee = p_first == 0 ? e : e - nt;
      int lo = 0, hi = 36;  // largest src with pre[src] <= ee
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (M.pre[mid] <= ee) lo = mid;
        else hi = mid;
      }
      srci_first = lo;
      const int sl = M.beg[lo] + (ee - M.pre[lo]);
      src_first = make_double4(__ldcg(T.sx + sl), __ldcg(T.sy + sl), __ldcg(T.sz + sl), __ldcg(T.sq + sl));
    }
    // window (src/energy_shift.cpp:72-90)
    for (int k = gtr; k < T.Hw; k += gstride) {
      const double2 t = phase_at(to.root, k, T.dw), o = phase_at(oo.root, k, T.dw);
      const double2 g = __ldcg(T.out_root + k);
      const double ar = t.x - o.x, ai = t.y - o.y, br = g.x - o.x, bi = g.y - o.y;
      acc[0] += (ar * br + ai * bi) * T.W[k];
    }
    // difference (src/energy_shift.cpp:92-140)
    {
      const int base = T.pw_base, d = T.dd;
      for (int k = gt; k < T.H; k += gstride) {
        const int ix = k % d, iy = (k / d) % d, iz = k / (d * d);
        double s = 0;
        for (int l = 2; l <= lo_max; ++l) {
          const double2 o = cmul(oo.lev[l][2][iz], cmul(oo.lev[l][1][iy], oo.lev[l][0][ix]));
          const double2 c = __ldcg(T.inc + size_t(h.path_o[l] - base) * T.H + k);
          s -= (o.x * c.x - o.y * c.y - (o.x * o.x + o.y * o.y)) * c_level[l];
        }
        for (int l = 2; l <= lt_max; ++l) {
          const double2 t = cmul(to.lev[l][2][iz], cmul(to.lev[l][1][iy], to.lev[l][0][ix]));
          const double2 c = __ldcg(T.inc + size_t(h.path_t[l] - base) * T.H + k);
          s += (t.x * c.x - t.y * c.y) * c_level[l];
        }
        acc[1] += s * T.D2[k];
      }
    }
    {
      for (; e < e1; e += blockDim.x) {
        int p, srci;
        double4 v;
        if (e == e0 + int(threadIdx.x)) {
          p = p_first;
          srci = srci_first;
          v = src_first;
        } else {
          p = e < nt ? 0 : 1;
          const ResMeta& M = meta[p];
          const int ee = p == 0 ? e : e - nt;
          int lo = 0, hi = 36;
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (M.pre[mid] <= ee) lo = mid;
            else hi = mid;
          }
          srci = lo;
          const int sl = M.beg[lo] + (ee - M.pre[lo]);
          v = make_double4(__ldcg(T.sx + sl), __ldcg(T.sy + sl), __ldcg(T.sz + sl), __ldcg(T.sq + sl));
        }
        const ResMeta& M = meta[p];
        const int lv = (p == 0 ? h.depth_t : h.depth_o) - 1;
        const double b = level_box(T, lv);
        const double* x = p == 0 ? h.xt : h.xo;
        const double dx = x[0] - (v.x + M.off[srci][0]), dy = x[1] - (v.y + M.off[srci][1]),
                     dz = x[2] - (v.z + M.off[srci][2]);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 > eps && r2 < b * b) acc[2 + p] += v.w * poly(sqrt(r2), b);
      }
      // arrivals parked in the overflow pool that belong to a source's subtree
      const int pn = s_pn;
      for (int e2 = gt; e2 < 2 * 36 * pn; e2 += gstride) {
        const int p = e2 / (36 * pn), sj = (e2 / pn) % 36, q = e2 % pn;
        const ResMeta& M = meta[p];
        if (M.cnt[sj] < 0 || __ldcg(T.p_orig + q) < 0) continue;
        const int pl = __ldcg(T.p_leaf + q);
        const int ll = T.node_level[pl], lj = M.lvl[sj];
        if (ll < lj || (T.node_prefix[pl] >> (3 * (ll - lj))) != M.pfx[sj]) continue;
        const int lv = (p == 0 ? h.depth_t : h.depth_o) - 1;
        const double b = level_box(T, lv);
        const double* x = p == 0 ? h.xt : h.xo;
        const double dx = x[0] - (__ldcg(T.px + q) + M.off[sj][0]), dy = x[1] - (__ldcg(T.py + q) + M.off[sj][1]),
                     dz = x[2] - (__ldcg(T.pz + q) + M.off[sj][2]);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 > eps && r2 < b * b) acc[2 + p] += __ldcg(T.pq + q) * poly(sqrt(r2), b);
      }
      acc[2] *= h.q;
      acc[3] *= h.q;
    }
    const int s_next = threadIdx.x < 32 ? __ldcg(T.orig_slot + i_next) : 0;
    block_sum4_t0(acc, red);
    double* part = a.partials + size_t(m & 1) * 4 * G;
    if (threadIdx.x == 0)
      for (int c = 0; c < 4; ++c) part[4 * blockIdx.x + c] = acc[c];
    if (!mc_barrier(T, a, nbar)) return;
    // every block reduces the same partials in the same order: one warp,
    // lane-strided sums then a shuffle tree into lane 0
    double tot[4] = {0, 0, 0, 0};
    if (threadIdx.x < 32) {
      for (int b = threadIdx.x; b < G; b += 32)
        for (int c = 0; c < 4; ++c) tot[c] += __ldcg(part + 4 * b + c);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        for (int o = 16; o > 0; o >>= 1) tot[c] += __shfl_down_sync(0xffffffffu, tot[c], o);
    }
    if (threadIdx.x == 0) {
      const double dEw = tot[0] * a.c_window;
      double self = 0;
      if (h.dr != 0) self = poly(h.dr, level_box(T, 2)) * h.q * h.q;
      const double dE = dEw + tot[1] + tot[2] - tot[3] - self;
      const int accd = a.u[m] < exp(-a.beta * dE) ? 1 : 0;
      s_acc = accd;
      if (blockIdx.x == 0) {
        if (a.dE_out) a.dE_out[m] = dE;
        if (a.acc_out) a.acc_out[m] = accd;
        // algorithmic bytes of the dE evaluation: root and incoming rows, W and
        // D, 32 B per near-field source particle
        const int nlev = max(lo_max - 1, 0) + max(lt_max - 1, 0);
        atomicAdd(&T.work[2], 24ull * T.Hw + 16ull * nlev * T.H + 8ull * T.H +
                                  32ull * (unsigned long long)(meta[0].pre[36] + meta[1].pre[36]));
      }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // the next particle's slot is stale when an accepted move changed leaves
      // (its own slot and the slot of the particle swapped into its place) or
      // moved that very particle
      const bool stale = s_acc && (h.path_o[h.depth_o - 1] != h.path_t[h.depth_t - 1] || i_next == h.i_orig);
      if (threadIdx.x == 0) s_stale = stale;
      // a kept slot is loaded now; an accepted move writes other slots only,
      // and the commit of a same-leaf move of this very particle marks it stale
      pre.s = -1;
      if (!stale) {
        pre.s = s_next;
        if (s_next < T.n_slots) {
          pre.x = __ldcg(T.sx + s_next);
          pre.y = __ldcg(T.sy + s_next);
          pre.z = __ldcg(T.sz + s_next);
          pre.q = __ldcg(T.sq + s_next);
        } else {
          const int pp = s_next - T.n_slots;
          pre.x = __ldcg(T.px + pp);
          pre.y = __ldcg(T.py + pp);
          pre.z = __ldcg(T.pz + pp);
          pre.q = __ldcg(T.pq + pp);
        }
      }
      i_cur = i_next;
      for (int c = 0; c < 3; ++c) d_cur[c] = d_next[c];
    }
    if (!s_acc) continue;
    // accept-and-update (src/tree.cpp:447-597)
    const int nr = build_receivers(T, h, rs);
    // receiver groups per mode: the g that minimises grid-stride rounds of
    // the H*g units times receivers per group
    int ng = 1;
    {
      int best = 1 << 30;
#pragma unroll
      for (int g = 1; g <= 8; ++g) {
        const int cost = s_rounds[g] * ((nr + g - 1) / g);
        if (cost < best) {
          best = cost;
          ng = g;
        }
      }
    }
    if (blockIdx.x == G / 2 && threadIdx.x == 0) {
      P.i_orig = h.i_orig;
      P.slot = h.slot;
      P.q = h.q;
      for (int c = 0; c < 3; ++c) {
        P.xo[c] = h.xo[c];
        P.xt[c] = h.xt[c];
      }
      P.depth_o = h.depth_o;
      P.depth_t = h.depth_t;
      for (int l = 0; l < MAXLV; ++l) {
        P.path_o[l] = l < h.depth_o ? h.path_o[l] : -1;
        P.path_t[l] = l < h.depth_t ? h.path_t[l] : -1;
      }
      P.accepted = 1;
      P.valid = 1;
      P.n_recv = nr;
      atomicAdd(&T.work[0], 1ull);
      atomicAdd(&T.work[1], 32ull * ((unsigned long long)T.Hw + (unsigned long long)nr * T.H));
      commit_move(T, P);
    }
    {
      // root window: out_root += t - o
      for (int k = gtr; k < T.Hw; k += gstride) {
        const double2 t = phase_at(to.root, k, T.dw), o = phase_at(oo.root, k, T.dw);
        double2 g = __ldcg(T.out_root + k);
        g = cadd(g, t);
        g = csub(g, o);
        T.out_root[k] = g;
      }
      // units (mode k, receiver group): a thread walks its group's receivers
      // in level runs. A periodic image multiplies a single-particle phase by
      // a cube root of unity w^-e, e = (k - n).f * 2^l mod 3, so each run
      // precomputes p, p w^-1, p w^-2 and a receiver only picks one.
      const int n = T.n_diff, d = T.dd;
      for (int u = gt; u < T.H * ng; u += gstride) {
        const int k = u % T.H, rg = u / T.H;
        const int r0 = (rg * nr) / ng, r1 = ((rg + 1) * nr) / ng;
        const int ix = k % d, iy = (k / d) % d, iz = k / (d * d);
        const int a0 = ((ix - n) % 3 + 3) % 3, a1 = ((iy - n) % 3 + 3) % 3, a2 = ((iz - n) % 3 + 3) % 3;
        int r = r0;
        while (r < r1) {
          const int l = rs[r].level;
          int re = r + 1;
          while (re < r1 && rs[re].level == l) ++re;
          const double2 pt0 = cmul(to.lev[l][2][iz], cmul(to.lev[l][1][iy], to.lev[l][0][ix]));
          const double2 po0 = cmul(oo.lev[l][2][iz], cmul(oo.lev[l][1][iy], oo.lev[l][0][ix]));
          const double2 pt1 = cmul(pt0, root6(-2)), pt2 = cmul(pt0, root6(-4));
          const double2 po1 = cmul(po0, root6(-2)), po2 = cmul(po0, root6(-4));
          const int two_l = (l & 1) ? 2 : 1;
          for (; r < re; r += UPD_UNROLL) {
            double2 v[UPD_UNROLL];
            size_t off[UPD_UNROLL];
#pragma unroll
            for (int q = 0; q < UPD_UNROLL; ++q) {
              if (r + q < re) {
                const Receiver& R = rs[r + q];
                off[q] = size_t(R.off) * T.H + k;
                v[q] = R.is_out ? __ldcg(T.out + off[q]) : __ldcg(T.inc + off[q]);
              }
            }
#pragma unroll
            for (int q = 0; q < UPD_UNROLL; ++q) {
              if (r + q < re) {
                const Receiver& R = rs[r + q];
                // the exponent sum lies in [-12, 12]
                const int et = ((a0 * R.ft[0] + a1 * R.ft[1] + a2 * R.ft[2]) * two_l + 12) % 3;
                const int eo = ((a0 * R.fo[0] + a1 * R.fo[1] + a2 * R.fo[2]) * two_l + 12) % 3;
                double2 del = make_double2(0.0, 0.0);
                if (R.has_t) del = et == 0 ? pt0 : (et == 1 ? pt1 : pt2);
                if (R.has_o) del = csub(del, eo == 0 ? po0 : (eo == 1 ? po1 : po2));
                if (R.is_out) T.out[off[q]] = cadd(v[q], del);
                else T.inc[off[q]] = make_double2(v[q].x + del.x, v[q].y - del.y);
              }
            }
          }
          r = re;
        }
      }
    }
    mc_arrive(a, nbar);
    pend = true;
  }
}

// ---------------------------------------------------------------------------
// Long Metropolis sequences. As k_mc, one cooperative launch with the whole
// move on every SM, and with the row updates deferred (see Pending), which
// leaves the chain of one move as the cost: k_mc spent 4.3 us in the resolve,
// 1.0-1.7 in the tables, 1.0 in the source lists, 2.1 in the decision and up
// to 2.6 waiting for the previous commit (N = 1e5, clock stamps). Here
//   - the warps of a block work side by side: difference modes, window modes,
//     near field, and a helper that resolves the next move (each block has a
//     fixed share of the modes, so a thread keeps its root coefficients and
//     table values in registers);
//   - a move's header, phase tables and source lists are made during the move
//     before it, the tables and lists while the block waits for the others'
//     sums; positions come from pos4, an array by particle that a move's commit
//     updates, so no slot is read and a particle swapped to another slot does
//     not matter. Only a particle moved twice in a row is resolved again;
//   - the blocks exchange one double each in a 16-byte packet {sum, epoch,
//     pool fill} that every block polls: arrival and data in one round trip;
//   - a commit writes the slots of two leaves, so the next move waits for it
//     only if one of them is among its sources (the exchange orders it for
//     every later move).
constexpr int MCL_T = 512, MCL_W = MCL_T / 32;
constexpr int MCL_UNITS = 16;   // pair units whose cosines are held at a time
constexpr int MCL_LEVB = 3;     // levels whose rows one thread loads together
constexpr int MCL_POLL = 5;     // packets a lane polls together

struct SrcList {
  int beg[36], end[36], leaf[36], lvl[36], cnt[36], pre[37];  // leaf: the node id of a leaf source, else -1; lvl -1: absent
  unsigned long long pfx[36];
  double off[36][3];
};

struct McLongArgs {
  const int* idx;
  const double* disp;
  const double* u;
  double beta;
  int n_moves;
  double* dE_out;
  int* acc_out;
  double c_window;
  unsigned long long* packets;  // [2][G][2], double-buffered by move parity, epochs cleared at launch
  unsigned int* committed;      // epoch of the last committed move
  double4* pos4;                // position and charge by particle, for the particles of this launch
  long long spin_limit;
  Pending* list;
  int* n_list;
  int* touched;
  const double* oct;
  int per_block;
};

template <int NP>
constexpr size_t mcl_bytes(int per_block) {
  using M = ModesOf<NP>;
  // the folded table in shared memory where it leaves room for deep trees' phase tables (n = 26: read through L1)
  return (M::ND <= 19 ? size_t(M::OCT) * 8 : 0) + size_t(MCL_UNITS) * M::CT * 8 + sizeof(Pending) * per_block +
         sizeof(int) * (MAXLV * per_block + 8);
}

__device__ inline void packet_store(unsigned long long* p, double v, unsigned epoch, unsigned extra) {
  const unsigned long long lo = (unsigned long long)__double_as_longlong(v);
  const unsigned long long hi = (unsigned long long)epoch | ((unsigned long long)extra << 32);
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
               "l"(lo), "l"(hi)
               : "memory");
}
__device__ inline void packet_load(const unsigned long long* p, double& v, unsigned& epoch, unsigned& extra) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  v = __longlong_as_double((long long)lo);
  epoch = unsigned(hi);
  extra = unsigned(hi >> 32);
}

// The same load once more as an acquire, for a packet that has arrived (it reads the
// same packet: the next one in its place waits for this block's own): what was
// released before the packet is visible after it. A fence behind the relaxed loads
// would order as much, for 800 cycles of every move; waiting for this load's value
// would take 0.3 us of the 8 of a move at N = 1e5.
__device__ inline void packet_acquire(const unsigned long long* p) {
  asm volatile("{\n .reg .b128 t;\n ld.acquire.gpu.global.b128 t, [%0];\n}\n" ::"l"(p) : "memory");
}

// positions and charges of the particles a launch will move
__global__ void k_gather_moves(DevTree T, const int* __restrict__ idx, int n, double4* pos4) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  const int i = idx[m], s = T.orig_slot[i], p = s - T.n_slots;
  pos4[i] = p < 0 ? make_double4(T.sx[s], T.sy[s], T.sz[s], T.sq[s]) : make_double4(T.px[p], T.py[p], T.pz[p], T.pq[p]);
}

// resolve() for one warp from a known position, the three bitmap words of a
// lane's level loaded together (bm, wp: the levels' bitmap and prefix pointers
// in shared memory)
__device__ __noinline__ void resolve_warp(const DevTree& T, int i, double4 at, double d0, double d1, double d2, Header& h,
                                          const uint32_t* const* bm, const int* const* wp) {
  const int lane = threadIdx.x & 31;
  const double L = T.L;
  const double xo[3] = {at.x, at.y, at.z};
  const double xt[3] = {wrap_mod(xo[0] + d0, L), wrap_mod(xo[1] + d1, L), wrap_mod(xo[2] + d2, L)};
  const int half = lane >> 4, l = lane & 15;
  const double* p = half == 0 ? xt : xo;
  const uint32_t g[3] = {grid_coord(p[0], L), grid_coord(p[1], L), grid_coord(p[2], L)};
  const uint64_t key = morton3(g[0], g[1], g[2]);
  const bool lv = l < T.max_depth;
  const uint64_t cell = l == 0 || !lv ? 0 : key >> (3 * (KEY_BITS - l));
  uint32_t w0 = 0, w1 = 0;
  int pr = 0;
  if (lv && l >= 2) {
    w0 = bm[l - 1][cell >> 8];
    pr = wp[l - 1][cell >> 8];
  }
  if (lv && l <= T.maxref) w1 = bm[l][cell >> 5];
  int node = -1;
  bool is_leaf = false;
  const unsigned c5 = unsigned(cell >> 3) & 31u;
  if (lv && (l <= 1 || ((w0 >> c5) & 1u))) {
    node = l == 0 ? 0 : (l == 1 ? 1 + int(cell) : T.level_start_d[l] + 8 * (pr + __popc(w0 & ((1u << c5) - 1u))) + int(cell & 7));
    is_leaf = !(l <= T.maxref && ((w1 >> (cell & 31)) & 1u));
  }
  const unsigned leaves = (__ballot_sync(0xffffffffu, is_leaf) >> (16 * half)) & 0xffffu;
  const int leaf_level = __ffs(leaves) - 1;
  if (l <= leaf_level) {
    int* path = half == 0 ? h.path_t : h.path_o;
    int(*X)[3] = half == 0 ? h.Xt : h.Xo;
    path[l] = node;
    for (int a = 0; a < 3; ++a) X[l][a] = int(g[a] >> (KEY_BITS - l));
  }
  if (lane == 0) {
    h.i_orig = i;
    h.q = at.w;
    for (int a = 0; a < 3; ++a) {
      h.xo[a] = xo[a];
      h.xt[a] = xt[a];
    }
    h.d2 = d0 * d0 + d1 * d1 + d2 * d2;
    h.depth_t = leaf_level + 1;
  }
  if (lane == 16) h.depth_o = leaf_level + 1;
  __syncwarp();
}

// res_meta without the leaf's current count
__device__ __noinline__ void source_static(const DevTree& T, int leaf, int l, const int* Xl, int src, SrcList& M) {
  const double b = level_box(T, l);
  int j = -1;
  if (src == 0) j = leaf;
  else if (src <= 27) j = (src - 1 == 13) ? -1 : T.col27[size_t(leaf) * 27 + (src - 1)];
  else j = T.coarse8[size_t(leaf) * 8 + (src - 28)];
  int beg = 0, end = 0, lj = -1, lf = -1;
  unsigned long long pj = 0;
  double off[3] = {0, 0, 0};
  if (j >= 0) {
    lj = T.node_level[j];
    pj = T.node_prefix[j];
    const int ch = T.node_child0[j];
    beg = T.node_begin[j];
    end = T.node_end[j];
    if (ch < 0) lf = j;
    const double bj = level_box(T, lj);
    const int Xj[3] = {int(compact3(pj)), int(compact3(pj >> 1)), int(compact3(pj >> 2))};
    for (int d = 0; d < 3; ++d)
      off[d] = -periodic_shift_d(center_of(T.L, l, Xl[d]), center_of(T.L, lj, Xj[d]), T.L, b, bj) * T.L;
  }
  M.beg[src] = beg;
  M.end[src] = end;
  M.leaf[src] = lf;
  M.lvl[src] = lj;
  M.pfx[src] = pj;
  for (int d = 0; d < 3; ++d) M.off[src][d] = off[d];
}

// build_tables with the mode counts known and the root box's spacing given
template <int NP>
__device__ __noinline__ void build_tables_of(const DevTree& T, const Header& h, int p, double2* tab, int t0, int nthr) {
  using MO = ModesOf<NP>;
  constexpr int nw = MO::NW, nd = MO::ND;
  constexpr int DW = 2 * nw + 1, D = 2 * nd + 1;
  constexpr int root_n = 2 * DW + nw + 1, lev_n = 2 * D + nd + 1;
  const double* x = p == 0 ? h.xo : h.xt;
  const int(*X)[3] = p == 0 ? h.Xo : h.Xt;
  const int lmax = (p == 0 ? h.depth_o : h.depth_t) - 2;
  const int total = root_n + (lmax >= 2 ? lmax - 1 : 0) * lev_n;
  for (int e = t0; e < total; e += nthr) {
    const bool root = e < root_n;
    const int l = root ? 0 : 2 + (e - root_n) / lev_n;
    const int rem = root ? e : (e - root_n) % lev_n;
    const int w = root ? DW : D;
    const int axis = rem < w ? 0 : (rem < 2 * w ? 1 : 2);
    const int t = rem - axis * w, m = t - (root ? nw : nd);
    const int Xa = root ? 0 : X[l][axis];
    const double xr = root ? x[axis] - 0.5 * T.L : x[axis] - center_of(T.L, l, Xa);
    const double th = (root ? T.delta_k[0] : level_dk(T, l)) * xr;
    const int dec = root ? 3 : 2 * Xa + 1;
    double2* dst = tab + (root ? axis * DW : 3 * DW + (l - 2) * 3 * D + axis * D);
    double sn, cs;
    sincos(-double(m) * th, &sn, &cs);
    const double sc = axis == 2 ? h.q : 1.0;
    dst[t] = cmul(make_double2(cs * sc, sn * sc), root6(-dec * m));
  }
}

__device__ inline void group_sync(int id, int n) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory"); }

template <int NP>
__global__ void __launch_bounds__(MCL_T, 1) k_mc_long(const __grid_constant__ DevTree T, McLongArgs a) {
  using MO = ModesOf<NP>;
  static_assert(MO::STR % 16 == 4 && MO::STR >= 8 * MO::MT, "bank layout");
  constexpr int D = 2 * MO::ND + 1, H = (MO::ND + 1) * D * D;
  constexpr int DW = 2 * MO::NW + 1, HW = (MO::NW + 1) * DW * DW;
  extern __shared__ double2 sm2[];
  // The chain of one move runs once through a lot of code: functions used in
  // several places are not inlined (they read the tree's description from
  // shared memory), so that the loop stays in the instruction caches.
  __shared__ __align__(16) unsigned char ts_raw[sizeof(DevTree)];
  __shared__ Header hb[3];
  __shared__ SrcList src[2][2];
  __shared__ double c_level[MAXLV + 2];
  __shared__ double red[MCL_W];
  __shared__ const uint32_t* s_bm[MAXLV];
  __shared__ const int* s_wp[MAXLV];
  __shared__ Proposal P;
  __shared__ double s_box[MAXLV], s_ibox[MAXLV];
  __shared__ int s_acc, s_ok, s_units, s_wait, s_pn, s_pool;
  const ResidualPoly<NP> poly(T);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const DevTree& Ts = *reinterpret_cast<const DevTree*>(ts_raw);
  for (int i = tid; i < int(sizeof(DevTree) / 4); i += MCL_T)
    reinterpret_cast<unsigned*>(ts_raw)[i] = reinterpret_cast<const unsigned*>(&T)[i];
  const int G = gridDim.x, B = blockIdx.x;
  // roles: warps [0, wd) difference modes, [wd, wd + ww) window modes, the
  // last the helper, the rest the near field. At most two modes a thread.
  const int hb0 = int(long(H) * B / G), hb1 = int(long(H) * (B + 1) / G);
  const int wb0 = int(long(HW) * B / G), wb1 = int(long(HW) * (B + 1) / G);
  const int wd = min(9, (H / G + 1 + 31) / 32), ww = min(3, (HW / G + 1 + 31) / 32);
  const int w_near = wd + ww;
  const bool commits = B == G / 2;  // the block that moves the particles, by its last near-field warp
  const int n_near = 32 * (MCL_W - 1 - w_near - (commits ? 1 : 0));
  const int dt = tid, wt = tid - 32 * wd, nt_ = tid - 32 * w_near;
  // phase tables of this move and the next, then the deferred-update part
  const int per = 3 * DW + max(T.max_depth - 1, 0) * 3 * D;
  double* dyn = reinterpret_cast<double*>(sm2 + 4 * per);
  const double* oct = a.oct;
  if (MO::ND <= 19) {
    for (int i = tid; i < MO::OCT; i += MCL_T) dyn[i] = a.oct[i];
    oct = dyn;
    dyn += MO::OCT;
  }
  double* ct = dyn;
  dyn += MCL_UNITS * MO::CT;
  Pending* mine = reinterpret_cast<Pending*>(dyn);
  int* act = reinterpret_cast<int*>(mine + a.per_block);
  int n_mine = 0, n_acc = 0;  // listed moves: this block's, all blocks'
  if (tid >= 2 && tid < MAXLV + 2) {
    const double dk = level_dk(T, tid);
    c_level[tid] = dk * dk * dk / (8.0 * 3.14159265358979323846 * 3.14159265358979323846 * 3.14159265358979323846) *
                   level_dscale(tid);
  }
  if (tid < MAXLV) {
    s_box[tid] = level_box(T, tid);
    s_ibox[tid] = 1.0 / s_box[tid];
  }
  if (tid < MAXLV && tid < T.max_depth) {
    s_bm[tid] = T.bm_d[tid];
    s_wp[tid] = T.wprefix_d[tid];
  }
  // this thread's modes: D2 and W values, root coefficients
  double tab_v[2] = {0.0, 0.0};
  double2 root_g[2] = {make_double2(0, 0), make_double2(0, 0)}, root_d[2];
  if (warp < wd) {
    for (int j = 0; j < 2; ++j)
      if (hb0 + dt + j * 32 * wd < hb1) tab_v[j] = T.D2[hb0 + dt + j * 32 * wd];
  } else if (warp < w_near) {
    for (int j = 0; j < 2; ++j)
      if (wb0 + wt + j * 32 * ww < wb1) {
        tab_v[j] = T.W[wb0 + wt + j * 32 * ww];
        root_g[j] = T.out_root[wb0 + wt + j * 32 * ww];
      }
  }
  unsigned long long work_de = 0;
  bool prev_acc = false;
  auto load_at = [&](int i) {
    const double* p = &a.pos4[i].x;
    return make_double4(__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3));
  };
  // the helper's next move and the index after it
  int nx_i = 0, nn_i = 0, prev_i = -1;
  double nx_d[3] = {0, 0, 0};
  double4 nx_at = make_double4(0, 0, 0, 0);
  auto tables_of = [&](int m, int p, Tables& tb) { alloc_tables(sm2 + ((m & 1) * 2 + p) * per, T, tb); };
  auto build_next = [&](int m, const Header& h, int t0, int nthr) {  // both paths' tables of move m
#pragma unroll 1
    for (int p = 0; p < 2; ++p) build_tables_of<NP>(Ts, h, p, sm2 + ((m & 1) * 2 + p) * per, t0, nthr);
  };
  // a leaf source's current count; a commit that changes it later makes the
  // near field count again
  auto count_source = [&](SrcList& M, int j) {
    M.cnt[j] = M.lvl[j] < 0 ? 0 : (M.leaf[j] >= 0 ? __ldcg(T.leaf_count + M.leaf[j]) : M.end[j] - M.beg[j]);
  };
  auto lists_next = [&](int m, const Header& h, int t) {  // source t of 72
    const int p = t / 36;
    const int lv = (p == 0 ? h.depth_t : h.depth_o) - 1;
    source_static(Ts, p == 0 ? h.path_t[lv] : h.path_o[lv], lv, p == 0 ? h.Xt[lv] : h.Xo[lv], t % 36, src[m & 1][p]);
    count_source(src[m & 1][p], t % 36);
  };
  // the rows of this block's modes go to L2 ahead of their use
  auto prefetch_rows = [&](const Header& h) {
    for (int p = 0; p < 2; ++p) {
      const int top = (p == 0 ? h.depth_t : h.depth_o) - 2;
      for (int l = 2; l <= top; ++l) {
        const double2* row = T.inc + size_t((p == 0 ? h.path_t[l] : h.path_o[l]) - T.pw_base) * H;
        for (int k = hb0 + 8 * lane; k < hb1; k += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + k));
      }
    }
  };
  if (tid == 0) s_pool = s_pn = __ldcg(T.pool_n);
  __syncthreads();
  if (warp == MCL_W - 1) {
    const int i = a.idx[0];
    resolve_warp(Ts, i, load_at(i), a.disp[0], a.disp[1], a.disp[2], hb[0], s_bm, s_wp);
    if (a.n_moves > 1) {
      nx_i = a.idx[1];
      nx_at = load_at(nx_i);
      for (int c = 0; c < 3; ++c) nx_d[c] = a.disp[3 + c];
    }
    if (a.n_moves > 2) nn_i = a.idx[2];
  }
  __syncthreads();
  build_next(0, hb[0], tid, MCL_T);
  if (tid < 72) lists_next(0, hb[0], tid);
  if (tid == 0) s_units = s_wait = 0;
  __syncthreads();

  for (int m = 0; m < a.n_moves; ++m) {
    const Header& h = hb[m % 3];
    Header& hn = hb[(m + 1) % 3];
    const bool more = m + 1 < a.n_moves;
    const unsigned epoch = unsigned(m) + 1u;
    Tables to, oo;
    tables_of(m, 0, oo);
    tables_of(m, 1, to);
    SrcList* S = src[m & 1];
    const int lo_max = h.depth_o - 2, lt_max = h.depth_t - 2;
    const double u_m = tid == 0 ? a.u[m] : 0.0;
    double v = 0.0;  // this thread's share of dE
    if (warp < wd) {
      // difference (src/energy_shift.cpp:92-140); the rows of MCL_LEVB levels
      // are loaded together, once where both paths share the box
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int k = hb0 + dt + j * 32 * wd;
        if (k < hb1) {
          const int ix = k % D, iy = (k / D) % D, iz = k / (D * D);
          const int top = max(lo_max, lt_max);
          double s = 0;
          for (int l0 = 2; l0 <= top; l0 += MCL_LEVB) {
            double2 co[MCL_LEVB], cn[MCL_LEVB];
#pragma unroll
            for (int q = 0; q < MCL_LEVB; ++q) {
              const int l = l0 + q;
              if (l <= lo_max) co[q] = __ldcg(T.inc + size_t(h.path_o[l] - T.pw_base) * H + k);
              if (l <= lt_max && !(l <= lo_max && h.path_o[l] == h.path_t[l]))
                cn[q] = __ldcg(T.inc + size_t(h.path_t[l] - T.pw_base) * H + k);
            }
#pragma unroll
            for (int q = 0; q < MCL_LEVB; ++q) {
              const int l = l0 + q;
              if (l <= lo_max) {
                const double2 o = cmul(oo.lev[l][2][iz], cmul(oo.lev[l][1][iy], oo.lev[l][0][ix]));
                s -= (o.x * co[q].x - o.y * co[q].y - (o.x * o.x + o.y * o.y)) * c_level[l];
              }
              if (l <= lt_max) {
                if (l <= lo_max && h.path_o[l] == h.path_t[l]) cn[q] = co[q];
                const double2 t = cmul(to.lev[l][2][iz], cmul(to.lev[l][1][iy], to.lev[l][0][ix]));
                s += (t.x * cn[q].x - t.y * cn[q].y) * c_level[l];
              }
            }
          }
          v += s * tab_v[j];
        }
      }
    } else if (warp < w_near) {
      // window (src/energy_shift.cpp:72-90)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int k = wb0 + wt + j * 32 * ww;
        if (k < wb1) {
          const double2 t = phase_at(to.root, k, DW), o = phase_at(oo.root, k, DW);
          const double2 g = root_g[j];
          root_d[j] = make_double2(t.x - o.x, t.y - o.y);
          v += (root_d[j].x * (g.x - o.x) + root_d[j].y * (g.y - o.y)) * tab_v[j];
        }
      }
      v *= a.c_window;
    } else if (nt_ < n_near) {
      // near field of the target and the origin (src/energy_shift.cpp:
      // 233-302): the pairs of both paths split evenly over the blocks
      if (s_wait) {  // the epoch of a commit that writes a leaf among the sources
        if (nt_ == 0) {
          int ok = 0;
          for (long long it = 0; it < a.spin_limit; ++it)
            if (ld_acquire(a.committed) >= unsigned(s_wait)) {
              ok = 1;
              break;
            }
          if (ok) s_pn = __ldcg(T.pool_n);
          else atomicOr(T.err, 2);
        }
        group_sync(1, n_near);
        for (int t = nt_; t < 72; t += n_near) count_source(S[t / 36], t % 36);
        group_sync(1, n_near);
      }
      if (nt_ < 64) {  // exclusive prefix of a path's 36 counts, one warp each
        SrcList& M = S[nt_ >> 5];
        int c0 = M.cnt[lane], c1 = lane < 4 ? M.cnt[32 + lane] : 0;
        int x = c0;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        const int tot = __shfl_sync(0xffffffffu, x, 31);
        int y1 = c1;
        for (int o = 1; o < 4; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, y1, o);
          if (lane >= o) y1 += y;
        }
        M.pre[lane] = x - c0;
        if (lane < 4) M.pre[32 + lane] = tot + y1 - c1;
        if (lane == 3) M.pre[36] = tot + y1;
      }
      group_sync(1, n_near);
      const int nt = S[0].pre[36], np = nt + S[1].pre[36];
      const int e0 = int((long(B) * np) / G), e1 = int((long(B + 1) * np) / G);
      const double eps = 2.220446049250313e-16;
      for (int e = e0 + nt_; e < e1; e += n_near) {
        const int p = e < nt ? 0 : 1;
        const SrcList& M = S[p];
        const int ee = p == 0 ? e : e - nt;
        int lo = 0, hi = 36;  // largest source with pre[] <= ee
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (M.pre[mid] <= ee) lo = mid;
          else hi = mid;
        }
        const int sl = M.beg[lo] + (ee - M.pre[lo]);
        const double4 w = make_double4(__ldcg(T.sx + sl), __ldcg(T.sy + sl), __ldcg(T.sz + sl), __ldcg(T.sq + sl));
        const int lv = (p == 0 ? h.depth_t : h.depth_o) - 1;
        const double b = s_box[lv];
        const double* x = p == 0 ? h.xt : h.xo;
        const double dx = x[0] - (w.x + M.off[lo][0]), dy = x[1] - (w.y + M.off[lo][1]), dz = x[2] - (w.z + M.off[lo][2]);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 > eps && r2 < b * b) {
          const double r = w.w * poly.from_r2_as_above(r2, b, s_ibox[lv]);
          v += p == 0 ? r : -r;
        }
      }
      // arrivals parked in the overflow pool that belong to a source's subtree:
      // every block takes its own range, since n_near is not the same in all of
      // them (the one that commits has a warp less)
      const int pn = s_pn;
      if (pn > 0) {
        const long n2 = 2L * 36 * pn;
        const int p0 = int(n2 * B / G), p1 = int(n2 * (B + 1) / G);
        for (int e2 = p0 + nt_; e2 < p1; e2 += n_near) {
          const int p = e2 / (36 * pn), sj = (e2 / pn) % 36, qi = e2 % pn;
          const SrcList& M = S[p];
          if (M.lvl[sj] < 0 || __ldcg(T.p_orig + qi) < 0) continue;
          const int pl = __ldcg(T.p_leaf + qi);
          const int ll = T.node_level[pl], lj = M.lvl[sj];
          if (ll < lj || (T.node_prefix[pl] >> (3 * (ll - lj))) != M.pfx[sj]) continue;
          const double b = level_box(T, (p == 0 ? h.depth_t : h.depth_o) - 1);
          const double* x = p == 0 ? h.xt : h.xo;
          const double dx = x[0] - (__ldcg(T.px + qi) + M.off[sj][0]), dy = x[1] - (__ldcg(T.py + qi) + M.off[sj][1]),
                       dz = x[2] - (__ldcg(T.pz + qi) + M.off[sj][2]);
          const double r2 = dx * dx + dy * dy + dz * dz;
          if (r2 > eps && r2 < b * b) {
            const double r = __ldcg(T.pq + qi) * poly(sqrt(r2), b);
            v += p == 0 ? r : -r;
          }
        }
      }
      v *= h.q;
    } else if (warp == MCL_W - 1 && more) {
      // helper: resolve the next move from what it loaded a move ago, and load
      // for the move after it. Of the commits that may have been running then,
      // the last move's position is in its header and the one before is in
      // pos4 by now
      const Header& hp = hb[(m + 2) % 3];  // move m - 1
      double4 at = nx_at;
      if (m > 1 && prev_i == nx_i) at = load_at(nx_i);
      if (m > 0 && hp.i_orig == nx_i && prev_acc) at = make_double4(hp.xt[0], hp.xt[1], hp.xt[2], hp.q);
      const int i = nx_i;
      const double d0 = nx_d[0], d1 = nx_d[1], d2 = nx_d[2];
      if (m > 0) prev_i = hp.i_orig;
      if (m + 2 < a.n_moves) {
        nx_i = nn_i;
        nx_at = load_at(nn_i);
        for (int c = 0; c < 3; ++c) nx_d[c] = a.disp[3 * size_t(m + 2) + c];
        if (m + 3 < a.n_moves) nn_i = a.idx[m + 3];
      }
      resolve_warp(Ts, i, at, d0, d1, d2, hn, s_bm, s_wp);
      prefetch_rows(hn);
    }
    // what the listed moves changed in the rows the difference sums read: the
    // mode warps, which are done before the near field
    if (warp < w_near) {
      const int nu = s_units;
      for (int u0 = 0; u0 < nu; u0 += MCL_UNITS) {
        const int n = min(MCL_UNITS, nu - u0);
        for (int w = warp; w < n; w += w_near) {
          const int unit = act[u0 + w];
          unit_cosines<MO::ND>(T.L, level_dk(T, unit & 15), h, mine[unit >> 8], unit, ct + w * MO::CT);
        }
        group_sync(2, 32 * w_near);
        for (int w = 0; w < n; w += 2) {
          const int ua = act[u0 + w], ub = act[u0 + min(w + 1, n - 1)];
          v += unit_pair_rows<MO::ND>(oct, ct + w * MO::CT, w + 1 < n, c_level[ua & 15] * h.q * mine[ua >> 8].q,
                                      c_level[ub & 15] * h.q * mine[ub >> 8].q, (warp + w) % w_near, w_near);
        }
        if (u0 + MCL_UNITS < nu) group_sync(2, 32 * w_near);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    unsigned long long* pk = a.packets + size_t(m & 1) * 2 * G;
    if (warp == 0) {
      // publish this block's sum, then gather everybody's in a fixed order
      double x = lane < MCL_W ? red[lane] : 0.0;
#pragma unroll
      for (int o = MCL_W / 2; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) {
        if (commits && prev_acc) asm volatile("fence.acq_rel.gpu;" ::: "memory");  // releases the commit since the last packet
        packet_store(pk + 2 * B, x, epoch, commits ? unsigned(s_pool) : 0u);
      }
      // the self term (src/energy_shift.cpp:30-41, one image per lane) while
      // the others' packets are on their way
      double dr2 = h.d2;
      if (lane < 27) {
        const int mx = lane % 3 - 1, my = (lane / 3) % 3 - 1, mz = lane / 9 - 1;
        const double ax = h.xt[0] - (h.xo[0] + mx * T.L), ay = h.xt[1] - (h.xo[1] + my * T.L),
                     az = h.xt[2] - (h.xo[2] + mz * T.L);
        dr2 = fmin(dr2, ax * ax + ay * ay + az * az);
      }
      for (int o = 16; o > 0; o >>= 1) dr2 = fmin(dr2, __shfl_xor_sync(0xffffffffu, dr2, o));
      const double self = dr2 > 0.0 ? poly.from_r2_as_above(dr2, s_box[2], s_ibox[2]) * h.q * h.q : 0.0;
      double tot = 0.0;
      bool ok = true;
      for (int b0 = 0; b0 < G; b0 += 32 * MCL_POLL) {
        double pv[MCL_POLL];
        unsigned px[MCL_POLL];
        for (long long it = 0;; ++it) {
          bool all = true;
#pragma unroll
          for (int j = 0; j < MCL_POLL; ++j) {
            const int b = b0 + lane + 32 * j;
            unsigned pe = epoch;
            pv[j] = 0.0;
            if (b < G) packet_load(pk + 2 * b, pv[j], pe, px[j]);
            all = all && pe == epoch;
          }
          if (all) break;
          if (it >= a.spin_limit || ((it & 1023) == 1023 && (ldm<true>(T.err) & 2))) {
            ok = false;
            break;
          }
        }
#pragma unroll
        for (int j = 0; j < MCL_POLL; ++j) {
          tot += pv[j];
          // the committing block's packet follows its fence: its commits so far
          // are visible from here on
          if (b0 + lane + 32 * j == G / 2) {
            s_pn = int(px[j]);
            packet_acquire(pk + 2 * (G / 2));
          }
        }
      }
      if (!ok) atomicOr(T.err, 2);
      ok = __all_sync(0xffffffffu, ok);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) tot += __shfl_down_sync(0xffffffffu, tot, o);
      if (lane == 0) {
        const double dE = tot - self;
        const int accd = u_m < exp(-a.beta * dE) ? 1 : 0;
        s_acc = accd;
        s_ok = ok;
        s_wait = 0;
        if (B == 0) {
          if (a.dE_out) a.dE_out[m] = dE;
          if (a.acc_out) a.acc_out[m] = accd;
          const int nlev = max(lo_max - 1, 0) + max(lt_max - 1, 0);
          work_de += 24ull * HW + 16ull * nlev * H + 8ull * H + 32ull * (unsigned long long)(S[0].pre[36] + S[1].pre[36]);
        }
      }
    } else if (more) {
      if (warp >= MCL_W - 3) {
        const int t = tid - 32 * (MCL_W - 3);
        if (t < 72) lists_next(m + 1, hn, t);
      } else {
        build_next(m + 1, hn, tid - 32, MCL_T - 128);
      }
    }
    __syncthreads();
    if (!s_ok) return;
    const bool accd = s_acc != 0;
    const bool again = accd && more && hn.i_orig == h.i_orig;  // resolved from the old position
    if (accd) {
      if (warp >= wd && warp < w_near) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int k = wb0 + wt + j * 32 * ww;
          if (k < wb1) {
            root_g[j] = cadd(root_g[j], root_d[j]);
            T.out_root[k] = root_g[j];
          }
        }
      }
      if (warp == 1 && n_acc % G == B) {
        // this block keeps the move, lists it for the end of the launch and
        // marks the outgoing rows it changes
        if (lane == 0) {
          fill_pending(T, h, mine[n_mine]);
          a.list[n_acc] = mine[n_mine];
        }
        for (int l = T.pw_lo + lane; l <= T.pw_hi; l += 32) {
          if (l <= h.depth_t - 1) atomicAdd(a.touched + (h.path_t[l] - T.pw_base), 1);
          if (l <= h.depth_o - 1) atomicAdd(a.touched + (h.path_o[l] - T.pw_base), 1);
        }
      }
      if (n_acc % G == B) ++n_mine;
      ++n_acc;
    }
    // Does this move's commit, or the last one's (the counts may be older),
    // write a leaf the next move reads? A source box on the move's target or
    // origin path holds that leaf.
    if (more && (accd || prev_acc) && warp >= 2 && warp < 5 && tid - 64 < 72) {
      const SrcList& M = src[(m + 1) & 1][(tid - 64) / 36];
      const int j = (tid - 64) % 36;
      const int l = M.lvl[j];
      auto holds = [&](const Header& g) {
        return (l < g.depth_t && morton3(g.Xt[l][0], g.Xt[l][1], g.Xt[l][2]) == M.pfx[j]) ||
               (l < g.depth_o && morton3(g.Xo[l][0], g.Xo[l][1], g.Xo[l][2]) == M.pfx[j]);
      };
      if (l >= 0 && ((accd && holds(h)) || (prev_acc && holds(hb[(m + 2) % 3])))) s_wait = accd ? int(epoch) : int(epoch) - 1;
    }
    if (again) {  // the particle just moved moves again: resolve it from where it is now
      __syncthreads();
      if (warp == MCL_W - 1) {
        const double4 at = make_double4(h.xt[0], h.xt[1], h.xt[2], h.q);
        double dn[3];
        for (int c = 0; c < 3; ++c) dn[c] = a.disp[3 * size_t(m + 1) + c];
        resolve_warp(Ts, h.i_orig, at, dn[0], dn[1], dn[2], hn, s_bm, s_wp);
      }
      __syncthreads();
      if (tid < 72) lists_next(m + 1, hn, tid);
      else build_next(m + 1, hn, tid - 72, MCL_T - 72);
      if (tid == 0) s_wait = int(epoch);
      __syncthreads();
    }
    if (more && warp == 1) {
      __syncwarp();
      const int nu = near_units(hn, mine, n_mine, act);
      if (lane == 0) s_units = nu;
    }
    prev_acc = accd;
    if (accd && commits && warp == MCL_W - 2 && lane == 0) {
      P.i_orig = h.i_orig;
      P.q = h.q;
      for (int c = 0; c < 3; ++c) {
        P.xo[c] = h.xo[c];
        P.xt[c] = h.xt[c];
      }
      P.depth_o = h.depth_o;
      P.depth_t = h.depth_t;
      for (int l = 0; l < MAXLV; ++l) {
        P.path_o[l] = l < h.depth_o ? h.path_o[l] : -1;
        P.path_t[l] = l < h.depth_t ? h.path_t[l] : -1;
      }
      P.accepted = 1;
      P.valid = 1;
      P.n_recv = 0;
    }
    __syncthreads();
    // the commit runs beside the next move's sums
    if (accd && commits && warp == MCL_W - 2 && lane == 0) {
      P.slot = __ldcg(T.orig_slot + P.i_orig);
      atomicAdd(&T.work[0], 1ull);
      atomicAdd(&T.work[1], 32ull * (unsigned long long)HW);
      if (commit_move(T, P)) a.pos4[P.i_orig] = make_double4(P.xt[0], P.xt[1], P.xt[2], P.q);
      s_pool = int(*(volatile int*)T.pool_n);
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.committed), "r"(epoch) : "memory");
    }
  }
  if (B == 0 && tid == 0) {
    *a.n_list = n_acc;
    atomicAdd(&T.work[2], work_de);
  }
}

// ---------------------------------------------------------------------------
// Replica sets: up to REP_CHUNK moves of many independent trees in one
// launch, one thread block per tree (the block resolves, sums, decides,
// updates and commits its tree's moves with block barriers only). Small
// replicas do not need a whole GPU per move, so running them side by side
// fills the SMs with independent work.
// Expansion updates are deferred as in k_mc_long: a block that updated its
// tree's rows move by move moved about 30 MB per accepted move through one SM
// (1.7 ms a move with 256 replicas; the whole set ran at 4.3 TB/s of DRAM).
constexpr int REP_T = 256;
constexpr int REP_CHUNK = 128;  // most moves between two updates of the rows
constexpr int REP_ILP = 4;      // modes a thread loads before it uses the first
constexpr int REP_UNITS = 8;    // pair units whose cosines are held at a time

template <int NP>
constexpr size_t rep_lazy_bytes() {
  using M = ModesOf<NP>;
  return (M::ND <= 19 ? size_t(M::OCT) * 8 : 0) + size_t(REP_UNITS) * M::CT * 8 +
         sizeof(int) * MAXLV * REP_CHUNK;
}

struct RepArgs {
  const DevTree* trees;
  int m, m0, cnt;       // moves per tree; this launch runs [m0, m0 + cnt)
  const int* idx;
  const double* disp;
  const double* u;
  double beta;
  double* dE_out;
  int* acc_out;
  const SequenceRows* rows;
};

template <int NP>
__global__ void __launch_bounds__(REP_T, 2) k_mc_rep(RepArgs a) {
  using MO = ModesOf<NP>;
  constexpr int D = 2 * MO::ND + 1, H = (MO::ND + 1) * D * D;
  constexpr int DW = 2 * MO::NW + 1, HW = (MO::NW + 1) * DW * DW;
  extern __shared__ double2 sm2[];
  __shared__ __align__(16) unsigned char ts_raw[sizeof(DevTree)];
  __shared__ Header h;
  __shared__ double red[4][32];
  __shared__ double c_level[MAXLV + 2];
  __shared__ Proposal P;
  __shared__ int s_acc, s_units;
  {
    const unsigned* src = reinterpret_cast<const unsigned*>(a.trees + blockIdx.x);
    unsigned* dst = reinterpret_cast<unsigned*>(ts_raw);
    for (int i = threadIdx.x; i < int(sizeof(DevTree) / 4); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const DevTree& T = *reinterpret_cast<const DevTree*>(ts_raw);
  const ResidualPoly<NP> poly(T);
  const double pi = 3.14159265358979323846;
  if (threadIdx.x >= 2 && threadIdx.x < MAXLV + 2) {
    const double dk = level_dk(T, threadIdx.x);
    c_level[threadIdx.x] = dk * dk * dk / (8.0 * pi * pi * pi) * level_dscale(threadIdx.x);
  }
  const double dk0 = T.delta_k[0];
  const double c_window = dk0 * dk0 * dk0 / (8.0 * pi * pi * pi);
  const SequenceRows rows = a.rows[blockIdx.x];
  Pending* list = rows.list;
  int* touched = rows.touched;
  const double* oct = rows.oct;
  double* dyn = reinterpret_cast<double*>(sm2 + 2 * (3 * DW + max(T.max_depth - 1, 0) * 3 * D));
  if (MO::ND <= 19) {
    for (int i = threadIdx.x; i < MO::OCT; i += blockDim.x) dyn[i] = oct[i];
    oct = dyn;
    dyn += MO::OCT;
  }
  double* ct = dyn;
  int* act = reinterpret_cast<int*>(dyn + REP_UNITS * MO::CT);
  int n_acc = 0;
  for (int mv = a.m0; mv < a.m0 + a.cnt; ++mv) {
    const size_t c = size_t(blockIdx.x) * a.m + mv;
    resolve(T, a.idx[c], a.disp + 3 * c, h);
    const int lo_max = h.depth_o - 2, lt_max = h.depth_t - 2;
    const int uo = min(h.depth_o - 1, T.pw_hi), ut = min(h.depth_t - 1, T.pw_hi);
    const int per = 3 * (2 * T.n_window + 1) + max(max(uo, ut) - 1, 0) * 3 * (2 * T.n_diff + 1);
    Tables to, oo;
    alloc_tables(sm2, T, oo);
    alloc_tables(sm2 + per, T, to);
    build_tables(T, h.xo, h.q, h.Xo, uo, oo, threadIdx.x, blockDim.x);
    build_tables(T, h.xt, h.q, h.Xt, ut, to, threadIdx.x, blockDim.x);
    __syncthreads();
    if (threadIdx.x < 32) {
      const int nu = near_units(h, list, n_acc, act);
      if (threadIdx.x == 0) s_units = nu;
    }
    double acc[4] = {0, 0, 0, 0};
    for (int k = threadIdx.x; k < HW; k += REP_T) {
      const double2 t = phase_at(to.root, k, DW), o = phase_at(oo.root, k, DW);
      const double2 g = T.out_root[k];
      const double ar = t.x - o.x, ai = t.y - o.y, br = g.x - o.x, bi = g.y - o.y;
      acc[0] += (ar * br + ai * bi) * T.W[k];
    }
    acc[1] = diff_sum<MO::ND, REP_T, REP_ILP>(T, h, oo, to, lo_max, lt_max, c_level);
    __syncthreads();
    // what the listed moves changed in the rows just read
    for (int u0 = 0; u0 < s_units; u0 += REP_UNITS) {
      const int n = min(REP_UNITS, s_units - u0), warp = threadIdx.x >> 5;
      if (warp < n) {
        const int unit = act[u0 + warp];
        unit_cosines<MO::ND>(T.L, level_dk(T, unit & 15), h, list[unit >> 8], unit, ct + warp * MO::CT);
      }
      __syncthreads();
      for (int w = 0; w < n; w += 2) {
        const int ua = act[u0 + w], ub = act[u0 + min(w + 1, n - 1)];
        acc[1] += unit_pair_rows<MO::ND>(oct, ct + w * MO::CT, w + 1 < n, c_level[ua & 15] * h.q * list[ua >> 8].q,
                                         c_level[ub & 15] * h.q * list[ub >> 8].q, warp, REP_T / 32);
      }
      __syncthreads();
    }
    const int lt = h.depth_t - 1, lo = h.depth_o - 1;
    acc[2] = residual_sum(T, poly, h.path_t[lt], lt, h.Xt[lt], h.xt);
    __syncthreads();  // the second call reuses the source-list arrays of the first
    acc[3] = residual_sum(T, poly, h.path_o[lo], lo, h.Xo[lo], h.xo);
    block_sum4(acc, red);
    if (threadIdx.x == 0) {
      double self = 0;
      if (h.dr != 0) self = poly(h.dr, level_box(T, 2)) * h.q * h.q;
      const double dE = acc[0] * c_window + acc[1] + (acc[2] - acc[3]) * h.q - self;
      const int accd = a.u[c] < exp(-a.beta * dE) ? 1 : 0;
      s_acc = accd;
      if (a.dE_out) a.dE_out[c] = dE;
      if (a.acc_out) a.acc_out[c] = accd;
    }
    __syncthreads();
    if (!s_acc) continue;
    // accept-and-update (src/tree.cpp:447-597) by this block: the root row,
    // the membership, and the move's turn in the list
    if (threadIdx.x == 0) {
      Pending e;
      fill_pending(T, h, e);
      list[n_acc] = e;
      for (int l = T.pw_lo; l <= e.u[0]; ++l) ++touched[h.path_t[l] - T.pw_base];
      for (int l = T.pw_lo; l <= e.u[1]; ++l) ++touched[h.path_o[l] - T.pw_base];
      P.i_orig = h.i_orig;
      P.slot = h.slot;
      P.q = h.q;
      for (int x = 0; x < 3; ++x) {
        P.xo[x] = h.xo[x];
        P.xt[x] = h.xt[x];
      }
      P.depth_o = h.depth_o;
      P.depth_t = h.depth_t;
      for (int l = 0; l < MAXLV; ++l) {
        P.path_o[l] = l < h.depth_o ? h.path_o[l] : -1;
        P.path_t[l] = l < h.depth_t ? h.path_t[l] : -1;
      }
      P.accepted = 1;
      P.valid = 1;
      P.n_recv = 0;
      atomicAdd(&T.work[0], 1ull);
      atomicAdd(&T.work[1], 32ull * (unsigned long long)T.Hw);
      commit_move(T, P);
    }
    ++n_acc;
    for (int k = threadIdx.x; k < HW; k += REP_T) {
      const double2 t = phase_at(to.root, k, DW), o = phase_at(oo.root, k, DW);
      T.out_root[k] = csub(cadd(T.out_root[k], t), o);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *rows.n_list = n_acc;
}

using McRepKernel = void (*)(RepArgs);
McRepKernel mc_rep_kernel(int np) {
  switch (np) {
    case 7: return k_mc_rep<7>;
    case 13: return k_mc_rep<13>;
    case 19: return k_mc_rep<19>;
    case 25: return k_mc_rep<25>;
    default: throw std::invalid_argument("unsupported residual polynomial");
  }
}

using McKernel = void (*)(DevTree, McArgs);
McKernel mc_kernel(int np) {
  switch (np) {
    case 7: return k_mc<7>;
    case 13: return k_mc<13>;
    case 19: return k_mc<19>;
    case 25: return k_mc<25>;
    default: throw std::invalid_argument("unsupported residual polynomial");
  }
}

using McLongKernel = void (*)(DevTree, McLongArgs);
McLongKernel mc_long_kernel(int np) {
  switch (np) {
    case 7: return k_mc_long<7>;
    case 13: return k_mc_long<13>;
    case 19: return k_mc_long<19>;
    case 25: return k_mc_long<25>;
    default: throw std::invalid_argument("unsupported residual polynomial");
  }
}

size_t mc_long_smem(int np, int per_block) {
  switch (np) {
    case 7: return mcl_bytes<7>(per_block);
    case 13: return mcl_bytes<13>(per_block);
    case 19: return mcl_bytes<19>(per_block);
    default: return mcl_bytes<25>(per_block);
  }
}

size_t rep_lazy_smem(int np) {
  switch (np) {
    case 7: return rep_lazy_bytes<7>();
    case 13: return rep_lazy_bytes<13>();
    case 19: return rep_lazy_bytes<19>();
    default: return rep_lazy_bytes<25>();
  }
}

// outgoing rows of the nodes the listed moves touched
void launch_flush_outgoing(const DevTree& D, const Pending* list, const int* n_list, const int* touched, cudaStream_t st) {
  const unsigned grid = unsigned(flush_blocks(D));
  switch (D.n_diff) {
    case 6: k_flush_outgoing<6><<<grid, FO_T, 0, st>>>(D, list, n_list, touched); break;
    case 12: k_flush_outgoing<12><<<grid, FO_T, 0, st>>>(D, list, n_list, touched); break;
    case 19: k_flush_outgoing<19><<<grid, FO_T, 0, st>>>(D, list, n_list, touched); break;
    case 26: k_flush_outgoing<26><<<grid, FO_T, 0, st>>>(D, list, n_list, touched); break;
    default: throw std::invalid_argument("unsupported mode count");
  }
  PDMK_LAUNCH_CHECK();
}

// the same for a set of trees; blocks: the largest flush_blocks of one
void launch_flush_set(int n_diff, const DevTree* trees, const SequenceRows* rows, int n_trees, int blocks, cudaStream_t st) {
  if (blocks == 0) return;
  const dim3 grid = set_grid(blocks, n_trees);
  switch (n_diff) {
    case 6: k_flush_set<6><<<grid, FO_T, 0, st>>>(trees, rows, n_trees); break;
    case 12: k_flush_set<12><<<grid, FO_T, 0, st>>>(trees, rows, n_trees); break;
    case 19: k_flush_set<19><<<grid, FO_T, 0, st>>>(trees, rows, n_trees); break;
    case 26: k_flush_set<26><<<grid, FO_T, 0, st>>>(trees, rows, n_trees); break;
    default: throw std::invalid_argument("unsupported mode count");
  }
  PDMK_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Many points against one state in one launch: candidate moves (k_shift_batch)
// and potentials (k_potential_batch). A block takes a group of GRP particles;
// with a point x on level-l box B its difference sum is
//   Re sum_k D(k) inc_B(k) exp(-i k.x)
//     = Re sum_{iz,iy} ez[iz] ey[iy] s(iz, iy),  s = sum_ix (D inc_B)[iz,iy,ix] ex[ix],
// so the inner sums are a matrix product of the row, lines (iz, iy) by columns
// ix, with the ex of all the group's points on B: FP64 tensor instructions
// (m8n8k4), whose A operand comes straight from global memory (each row is
// read once for all its points) and whose cost per mode and point is the four
// multiply-adds of s. The thread-per-mode form took a product of three phases
// for every mode and point (10 operations, 12 shared-memory wavefronts per 32
// modes) and every candidate read its rows alone: 4096 candidates at N = 1e6
// moved 13.6 GB through L2 in 2.35 ms. Groups are formed along the Morton
// order of the particles (k_order_particles), so most of a group's points
// share their boxes; the result of a point does not depend on its group.
constexpr int BG_T = 256, BG_W = BG_T / 32;

template <int NP>
struct BatchShape {
  using MO = ModesOf<NP>;
  static constexpr int N1 = MO::ND + 1, D = 2 * MO::ND + 1, H = N1 * D * D;
  static constexpr int DW = 2 * MO::NW + 1, HW = (MO::NW + 1) * DW * DW;
  static constexpr int LINES = N1 * D, MT = (LINES + 7) / 8, KS = (D + 3) / 4;
  // D over the octant (|kz|, |ky|, |kx|) in shared memory where it fits; the
  // row stride is 4 or 12 modulo 16, so that 4 lines x 4 kx fall on different banks
  static constexpr bool TAB = MO::ND <= 19;
  static constexpr int DS = N1 % 16 <= 4 ? N1 / 16 * 16 + 4 : N1 % 16 <= 12 ? N1 / 16 * 16 + 12 : N1 / 16 * 16 + 20;
  static constexpr int TAB_DOUBLES = TAB ? N1 * N1 * DS : 0;
  __host__ __device__ static int per(int max_depth) { return 3 * DW + (max_depth > 3 ? max_depth - 3 : 0) * 3 * D; }  // phases of one point
  static size_t smem(int max_depth, int points) {
    return sizeof(double) * TAB_DOUBLES + sizeof(double2) * size_t(per(max_depth)) * points;
  }
};

// The points of a group and, per level, their distinct boxes
template <int PTS>
struct BatchRows {
  int n[MAXLV];                 // distinct boxes of a level
  int row[MAXLV][PTS];          // their expansion rows
  unsigned char npt[MAXLV][PTS];
  unsigned char pt[MAXLV][PTS][PTS];  // the points on each
};

// one thread: the rows of points 0 .. PTS-1 (node_of(p, l) < 0: the point has no box at level l)
template <int PTS, class F>
__device__ void batch_rows(BatchRows<PTS>& R, int top, F node_of) {
  for (int l = 2; l <= top; ++l) {
    int n = 0;
    for (int p = 0; p < PTS; ++p) {
      const int row = node_of(p, l);
      if (row < 0) continue;
      int r = 0;
      while (r < n && R.row[l][r] != row) ++r;
      if (r == n) {
        R.row[l][r] = row;
        R.npt[l][r] = 0;
        ++n;
      }
      R.pt[l][r][R.npt[l][r]++] = static_cast<unsigned char>(p);
    }
    R.n[l] = n;
  }
}

template <int NP>
__device__ void load_octant(const DevTree& T, double* tab) {
  using S = BatchShape<NP>;
  if constexpr (S::TAB)
#pragma unroll 8
    for (int i = threadIdx.x; i < S::TAB_DOUBLES; i += BG_T) {
      const int mx = i % S::DS, r = i / S::DS, mz = r / S::N1, my = r % S::N1;
      tab[i] = mx < S::N1 ? T.D2[((S::N1 - 1 - mz) * S::D + S::N1 - 1 + my) * S::D + S::N1 - 1 + mx] : 0.0;
    }
}

// The products of one row with the columns of up to NT tiles. COLS columns per
// point: 2 (re, im of ex), or 4 (and those of kx ex, in units of dk). consume(tile,
// line, c0, c1): this lane's two results, the (re, im) of its column pair (lane
// & 3) on its line.
template <int NP, int NT, int COLS, class F>
__device__ __forceinline__ void row_products(const DevTree& T, const double2* __restrict__ row, const double* __restrict__ tab,
                                             const double2* const (&ex)[NT], F consume) {
  using S = BatchShape<NP>;
  constexpr int KS = S::KS, D = S::D, ND = S::N1 - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q4 = lane & 3, q8 = lane >> 2;
  // B: this lane's column (lane >> 2) at ix = 4 s + (lane & 3), for the real
  // and the imaginary part of the row
  double bre[NT][KS], bim[NT][KS];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const int ix = 4 * k + q4;
      double2 v = make_double2(0.0, 0.0);
      if (ix < D && ex[t]) v = ex[t][ix];
      if (COLS == 4 && (q8 & 2)) v = cscale(v, double(ix - ND));
      bre[t][k] = (q8 & 1) ? v.y : v.x;
      bim[t][k] = (q8 & 1) ? v.x : -v.y;
    }
  for (int mt = warp; mt < S::MT; mt += BG_W) {
    const int line = min(8 * mt + q8, S::LINES - 1);
    const int iy = line % D, iz = line / D;
    const double2* src = row + size_t(line) * D + q4;
    double2 a[KS];
#pragma unroll
    for (int k = 0; k < KS; ++k) a[k] = 4 * k + q4 < D ? src[4 * k] : make_double2(0.0, 0.0);
    double c[NT][2][2];  // [row real, imaginary][column pair]
#pragma unroll
    for (int t = 0; t < NT; ++t) c[t][0][0] = c[t][0][1] = c[t][1][0] = c[t][1][1] = 0.0;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const int ix = 4 * k + q4;
      double d = 0.0;
      if (ix < D) d = S::TAB ? tab[((ND - iz) * S::N1 + abs(iy - ND)) * S::DS + abs(ix - ND)] : T.D2[size_t(line) * D + ix];
      const double ar = a[k].x * d, ai = a[k].y * d;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
            : "+d"(c[t][0][0]), "+d"(c[t][0][1])
            : "d"(ar), "d"(bre[t][k]));
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
            : "+d"(c[t][1][0]), "+d"(c[t][1][1])
            : "d"(ai), "d"(bim[t][k]));
      }
    }
    if (8 * mt + q8 < S::LINES)
#pragma unroll
      for (int t = 0; t < NT; ++t) consume(t, iz, iy, make_double2(c[t][0][0] + c[t][1][0], c[t][0][1] + c[t][1][1]));
  }
}

// source lists of a group's points (36 per point) with their prefix sums
template <int PTS>
struct BatchSources {
  int beg[PTS][36], pre[PTS][37], lvl[PTS][36];
  unsigned long long pfx[PTS][36];
  double off[PTS][36][3];
};

// block-cooperative; leaf(p), level(p) and X(p) give a point's leaf (level < 0: no point)
template <int PTS, class F>
__device__ void batch_sources(const DevTree& T, BatchSources<PTS>& S, F point) {
  for (int t = threadIdx.x; t < PTS * 36; t += BG_T) {
    const int p = t / 36, src = t % 36;
    int leaf, l;
    const int* Xl;
    point(p, leaf, l, Xl);
    int j = -1;
    if (l >= 0) {
      if (src == 0) j = leaf;
      else if (src <= 27) j = (src - 1 == 13) ? -1 : T.col27[size_t(leaf) * 27 + (src - 1)];
      else j = T.coarse8[size_t(leaf) * 8 + (src - 28)];
    }
    int beg = 0, cnt = 0, lj = -1;
    unsigned long long pj = 0;
    double off[3] = {0, 0, 0};
    if (j >= 0) {
      lj = T.node_level[j];
      pj = T.node_prefix[j];
      beg = T.node_begin[j];
      cnt = T.node_child0[j] < 0 ? T.leaf_count[j] : T.node_end[j] - beg;
      const double b = level_box(T, l), bj = level_box(T, lj);
      const int Xj[3] = {int(compact3(pj)), int(compact3(pj >> 1)), int(compact3(pj >> 2))};
      for (int d = 0; d < 3; ++d)
        off[d] = -periodic_shift_d(center_of(T.L, l, Xl[d]), center_of(T.L, lj, Xj[d]), T.L, b, bj) * T.L;
    }
    S.beg[p][src] = beg;
    S.pre[p][src] = cnt;
    S.lvl[p][src] = lj;
    S.pfx[p][src] = pj;
    for (int d = 0; d < 3; ++d) S.off[p][src][d] = off[d];
  }
  __syncthreads();
  if (threadIdx.x < PTS) {
    int s = 0;
    for (int src = 0; src < 36; ++src) {
      const int n = S.pre[threadIdx.x][src];
      S.pre[threadIdx.x][src] = s;
      s += n;
    }
    S.pre[threadIdx.x][36] = s;
  }
  __syncthreads();
}

// this thread's share of a point's near-field pairs: f(q_j, dx, dy, dz, r2) for
// each within the cut-off, overflow pool included
template <int PTS, class F>
__device__ __forceinline__ void batch_near(const DevTree& T, const BatchSources<PTS>& S, int p, const double* x, double b,
                                           int pool_n, F f) {
  const double eps = 2.220446049250313e-16, b2 = b * b;
  int src = 0;
  const int total = S.pre[p][36];
  for (int e = threadIdx.x; e < total; e += BG_T) {
    while (e >= S.pre[p][src + 1]) ++src;
    const int s = S.beg[p][src] + (e - S.pre[p][src]);
    const double dx = x[0] - (T.sx[s] + S.off[p][src][0]), dy = x[1] - (T.sy[s] + S.off[p][src][1]),
                 dz = x[2] - (T.sz[s] + S.off[p][src][2]);
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > eps && r2 < b2) f(T.sq[s], dx, dy, dz, r2);
  }
  for (int e = threadIdx.x; e < 36 * pool_n; e += BG_T) {
    const int sj = e / pool_n, q = e % pool_n;
    if (S.lvl[p][sj] < 0 || T.p_orig[q] < 0) continue;
    const int pl = T.p_leaf[q];
    const int ll = T.node_level[pl], lj = S.lvl[p][sj];
    if (ll < lj || (T.node_prefix[pl] >> (3 * (ll - lj))) != S.pfx[p][sj]) continue;
    const double dx = x[0] - (T.px[q] + S.off[p][sj][0]), dy = x[1] - (T.py[q] + S.off[p][sj][1]),
                 dz = x[2] - (T.pz[q] + S.off[p][sj][2]);
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > eps && r2 < b2) f(T.pq[q], dx, dy, dz, r2);
  }
}

// sums of N values over the block, the results in every thread
template <int N>
__device__ void batch_block_sum(double (&v)[N], double (*sm)[BG_W]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i)
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < N; ++i) sm[i][warp] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    double s = 0;
    for (int w = 0; w < BG_W; ++w) s += sm[i][w];
    v[i] = s;
  }
}

// GRP = 2: pairs along the Morton order where there are enough particles to
// fill the SMs, else one particle a block. (Groups of 4 read a third less, but their
// columns leave room for one block per SM: 1.43 against 1.12 ms for 4096 candidates.)
constexpr int BG_GROUP = 2;
// two groups of two per SM and residency; in pairs / one by one, us (N = 1e6, 9
// digits, host arrays): candidates 438 / 394 for 888, 502 / 508 for 1184, 634 /
// 679 for 1776; potentials 330 / 336, 353 / 414, 478 / 583
constexpr int kGroupMin = 4 * 148 * 2;
// At 3 digits (7 coefficients) a row is 19 KB and the work between two barriers so
// small that more resident blocks are worth more than shared rows: four a SM, one
// point each. 4096 candidates / potentials, us: N = 1e6 196 / 244 (in pairs at two
// blocks a SM 292 / 315, a thread per mode 238 / 311), N = 128e3 157 / 208 (214 /
// 253, 175 / 255).
__host__ __device__ constexpr int batch_blocks(int np) { return np == 7 ? 4 : 2; }
constexpr bool in_pairs(int np, int m) { return np > 7 && m >= kGroupMin; }

// order[]: the particles idx[0 .. m) by the level-4 cell of their positions (one
// block; the order within a cell is free, no result depends on it)
__global__ void __launch_bounds__(1024) k_order_particles(DevTree T, const int* __restrict__ idx, int m,
                                                          int* __restrict__ order) {
  __shared__ int bin[4096];
  __shared__ int wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto key = [&](int c) {
    const int s = T.orig_slot[idx[c]], p = s - T.n_slots;
    const double x = p < 0 ? T.sx[s] : T.px[p], y = p < 0 ? T.sy[s] : T.py[p], z = p < 0 ? T.sz[s] : T.pz[p];
    return int(morton3(grid_coord(x, T.L), grid_coord(y, T.L), grid_coord(z, T.L)) >> (3 * (KEY_BITS - 4)));
  };
  for (int i = threadIdx.x; i < 4096; i += 1024) bin[i] = 0;
  __syncthreads();
  for (int c = threadIdx.x; c < m; c += 1024) atomicAdd(&bin[key(c)], 1);
  __syncthreads();
  int v[4], sum = 0;
  for (int k = 0; k < 4; ++k) {
    v[k] = bin[4 * threadIdx.x + k];
    sum += v[k];
  }
  int x = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int at = (warp > 0 ? wsum[warp - 1] : 0) + x - sum;
  for (int k = 0; k < 4; ++k) {
    bin[4 * threadIdx.x + k] = at;
    at += v[k];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < m; c += 1024) order[atomicAdd(&bin[key(c)], 1)] = c;
}

template <int NP, int GRP>
__global__ void __launch_bounds__(BG_T, batch_blocks(NP)) k_shift_batch(DevTree T, const int* __restrict__ idx,
                                                      const double* __restrict__ disp, const int* __restrict__ order, int m,
                                                      double c_window, double sum_d2, double* __restrict__ dE_out) {
  using S = BatchShape<NP>;
  constexpr int PTS = 2 * GRP, NT = (PTS + 3) / 4;  // point 2 g: target of candidate g, 2 g + 1: its origin
  extern __shared__ double sm_b[];
  __shared__ Header hs[GRP];
  __shared__ BatchRows<PTS> rows;
  __shared__ BatchSources<PTS> srcs;
  __shared__ double red[PTS > 4 ? PTS : 4][BG_W];
  __shared__ double c_level[MAXLV + 2];
  const ResidualPoly<NP> poly(T);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q4 = lane & 3;
  double* tab = sm_b;
  double2* phases = reinterpret_cast<double2*>(sm_b + S::TAB_DOUBLES);
  const int per = S::per(T.max_depth);
  const int n = min(GRP, m - int(blockIdx.x) * GRP);
  if (tid >= 2 && tid < MAXLV + 2) {
    const double dk = level_dk(T, tid);
    c_level[tid] = dk * dk * dk / (8.0 * 3.14159265358979323846 * 3.14159265358979323846 * 3.14159265358979323846) *
                   level_dscale(tid);
  }
  int cand[GRP];
#pragma unroll
  for (int g = 0; g < GRP; ++g) {
    const int at = blockIdx.x * GRP + min(g, n - 1);
    cand[g] = order ? order[at] : at;
  }
#pragma unroll
  for (int g = 0; g < GRP; ++g)
    if (warp == g) resolve_by_warp(T, idx[cand[g]], disp + 3 * size_t(cand[g]), hs[g]);
  load_octant<NP>(T, tab);
  __syncthreads();
  int top = 0;
  for (int g = 0; g < n; ++g) top = max(top, max(hs[g].depth_o, hs[g].depth_t) - 2);
  if (tid == 0)
    batch_rows<PTS>(rows, top, [&](int p, int l) {
      const Header& h = hs[p >> 1];
      const int last = ((p & 1) ? h.depth_o : h.depth_t) - 2;
      if ((p >> 1) >= n || l > last) return -1;
      return ((p & 1) ? h.path_o[l] : h.path_t[l]) - T.pw_base;
    });
  for (int p = 0; p < 2 * n; ++p) {
    const Header& h = hs[p >> 1];
    Tables tb;
    alloc_tables(phases + size_t(p) * per, T, tb);
    if (p & 1) build_tables(T, h.xo, h.q, h.Xo, h.depth_o - 2, tb, tid, BG_T);
    else build_tables(T, h.xt, h.q, h.Xt, h.depth_t - 2, tb, tid, BG_T);
  }
  batch_sources<PTS>(T, srcs, [&](int p, int& leaf, int& l, const int*& Xl) {
    const Header& h = hs[p >> 1];
    l = (p >> 1) < n ? ((p & 1) ? h.depth_o : h.depth_t) - 1 : -1;
    if (l < 0) return;
    leaf = (p & 1) ? h.path_o[l] : h.path_t[l];
    Xl = (p & 1) ? h.Xo[l] : h.Xt[l];
  });
  // window (src/energy_shift.cpp:72-90)
  double v[GRP];
#pragma unroll
  for (int g = 0; g < GRP; ++g) v[g] = 0.0;
  for (int k = tid; k < S::HW; k += BG_T) {
    const double2 g0 = T.out_root[k];
    const double w = T.W[k];
#pragma unroll
    for (int g = 0; g < GRP; ++g) {
      if (g < n) {
        Tables to, oo;
        alloc_tables(phases + size_t(2 * g) * per, T, to);
        alloc_tables(phases + size_t(2 * g + 1) * per, T, oo);
        const double2 t = phase_at(to.root, k, S::DW), o = phase_at(oo.root, k, S::DW);
        v[g] += ((t.x - o.x) * (g0.x - o.x) + (t.y - o.y) * (g0.y - o.y)) * w;
      }
    }
  }
#pragma unroll
  for (int g = 0; g < GRP; ++g) v[g] *= c_window;
  // near field (src/energy_shift.cpp:233-302)
  const int pool_n = *T.pool_n;
#pragma unroll
  for (int g = 0; g < GRP; ++g) {
    if (g < n) {
      const Header& h = hs[g];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const double b = level_box(T, (p ? h.depth_o : h.depth_t) - 1);
        double a = 0.0;
        batch_near<PTS>(T, srcs, 2 * g + p, p ? h.xo : h.xt, b, pool_n,
                        [&](double q, double, double, double, double r2) { a += q * poly(sqrt(r2), b); });
        v[g] += (p ? -a : a) * h.q;
      }
    }
  }
  // difference (src/energy_shift.cpp:92-140), row by row; a warp's sums of a
  // point add up over the levels in its own words
  if (lane < PTS) red[lane][warp] = 0.0;
  __syncwarp();
  for (int l = 2; l <= top; ++l)
    for (int r = 0; r < rows.n[l]; ++r) {
      const double2* row = T.inc + size_t(rows.row[l][r]) * S::H;
      const int np = rows.npt[l][r];
      const unsigned char* pts = rows.pt[l][r];
      auto run = [&](auto nt) {
        constexpr int N = decltype(nt)::value;
        const double2* ex[N];
        const double2 *ey[N], *ez[N];
        double acc[N];
#pragma unroll
        for (int t = 0; t < N; ++t) {
          const int jb = 4 * t + (lane >> 3), jc = 4 * t + q4;  // the points of this lane's B column and results
          auto lev = [&](int j, int ax) {
            return phases + size_t(pts[min(j, np - 1)]) * per + 3 * S::DW + (l - 2) * 3 * S::D + ax * S::D;
          };
          ex[t] = jb < np ? lev(jb, 0) : nullptr;
          ey[t] = lev(jc, 1);
          ez[t] = lev(jc, 2);
          acc[t] = 0.0;
        }
        row_products<NP, N, 2>(T, row, tab, ex, [&](int t, int iz, int iy, double2 sv) {
          const double2 pz = cmul(ez[t][iz], ey[t][iy]);
          acc[t] += pz.x * sv.x - pz.y * sv.y;
        });
#pragma unroll
        for (int t = 0; t < N; ++t) {
          for (int o = 4; o < 32; o <<= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
          const int j = 4 * t + lane;
          if (lane < 4 && j < np) red[pts[j]][warp] += ((pts[j] & 1) ? -c_level[l] : c_level[l]) * acc[t];
        }
        __syncwarp();
      };
      if (NT > 1 && np > 4) run(std::integral_constant<int, NT>{});
      else run(std::integral_constant<int, 1>{});
    }
  // totals: one thread per candidate adds its points' words of all warps
  __syncthreads();
  double diff = 0.0;
  if (tid < n)
    for (int p = 0; p < 2; ++p)
      for (int w = 0; w < BG_W; ++w) diff += red[2 * tid + p][w];
  batch_block_sum<GRP>(v, red);
  if (tid < n) {
    const Header& h = hs[tid];
    double tot = 0.0;
#pragma unroll
    for (int g = 0; g < GRP; ++g)
      if (g == tid) tot = v[g];
    for (int l = 2; l <= h.depth_o - 2; ++l) diff += c_level[l] * h.q * h.q * sum_d2;  // |o|^2 = q^2 at every mode
    double self = 0;
    if (h.dr != 0) self = poly(h.dr, level_box(T, 2)) * h.q * h.q;
    int c = 0;
#pragma unroll
    for (int g = 0; g < GRP; ++g)
      if (g == tid) c = cand[g];
    dE_out[c] = tot + diff - self;
  }
}

using ShiftBatchKernel = void (*)(DevTree, const int*, const double*, const int*, int, double, double, double*);
ShiftBatchKernel shift_batch_kernel(int np, int grp) {
  switch (np) {
    case 7: return k_shift_batch<7, 1>;
    case 13: return grp > 1 ? k_shift_batch<13, BG_GROUP> : k_shift_batch<13, 1>;
    case 19: return grp > 1 ? k_shift_batch<19, BG_GROUP> : k_shift_batch<19, 1>;
    case 25: return grp > 1 ? k_shift_batch<25, BG_GROUP> : k_shift_batch<25, 1>;
    default: throw std::invalid_argument("unsupported residual polynomial");
  }
}

// shared memory of a batch kernel with `points` points a block
size_t batch_smem(int np, int max_depth, int points) {
  switch (np) {
    case 7: return BatchShape<7>::smem(max_depth, points);
    case 13: return BatchShape<13>::smem(max_depth, points);
    case 19: return BatchShape<19>::smem(max_depth, points);
    default: return BatchShape<25>::smem(max_depth, points);
  }
}

// ---------------------------------------------------------------------------
// Potential and field at particles: the same terms as an energy shift, for the
// particles' own positions only. With unit-charge phases u(k) = exp(-i k.x) and
// the particle's charge q, the interaction with all other particles is
//   c_w sum_{k != 0} W Re(u conj(g - q u)) + sum_l c_l sum_k D (Re(u inc_l) - q |u|^2)
//       + sum_{j != i} q_j res(r_ij),
// and the returned potential adds 2 q C, C the particle's self terms of the
// energy (window: c_w/2 sum W - psi0(0)/(2 bs_2 C0); each difference level on
// its path: c_l/2 sum D_l - S_l), so that E = 1/2 sum_i q_i phi_i and
// phi_i = dE/dq_i. The field is -grad phi, each plane wave differentiating to
// -i k u: the row products carry two more columns per point, kx ex, and the y
// and z derivatives take their factors at the lines.
template <int NP, int GRP>
__global__ void __launch_bounds__(BG_T, batch_blocks(NP)) k_potential_batch(DevTree T, const int* __restrict__ idx,
                                                          const int* __restrict__ order, int m, double c_window,
                                                          double self_w, double sum_w, double sum_d2,
                                                          const double* __restrict__ Sl,
                                                          double* __restrict__ phi_out, double* __restrict__ field_out) {
  using S = BatchShape<NP>;
  constexpr int ND = S::N1 - 1, NW = (S::DW - 1) / 2, NT = (GRP + 1) / 2;
  extern __shared__ double sm_b[];
  __shared__ Header hs[GRP];
  __shared__ BatchRows<GRP> rows;
  __shared__ BatchSources<GRP> srcs;
  __shared__ double red[4][BG_W];
  __shared__ double dsum[GRP][4][BG_W];  // difference part: phi, gradient
  __shared__ double c_level[MAXLV + 2];
  const ResidualPoly<NP> poly(T);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q4 = lane & 3;
  double* tab = sm_b;
  double2* phases = reinterpret_cast<double2*>(sm_b + S::TAB_DOUBLES);
  const int per = S::per(T.max_depth);
  const int n = min(GRP, m - int(blockIdx.x) * GRP);
  if (tid >= 2 && tid < MAXLV + 2) {
    const double dk = level_dk(T, tid);
    c_level[tid] = dk * dk * dk / (8.0 * 3.14159265358979323846 * 3.14159265358979323846 * 3.14159265358979323846) *
                   level_dscale(tid);
  }
  int cand[GRP];
#pragma unroll
  for (int g = 0; g < GRP; ++g) {
    const int at = blockIdx.x * GRP + min(g, n - 1);
    cand[g] = order ? order[at] : at;
  }
  const double zero3[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int g = 0; g < GRP; ++g)
    if (warp == g) resolve_by_warp(T, idx[cand[g]], zero3, hs[g]);
  load_octant<NP>(T, tab);
  __syncthreads();
  int top = 0;
  for (int g = 0; g < n; ++g) top = max(top, hs[g].depth_o - 2);
  if (tid == 0)
    batch_rows<GRP>(rows, top, [&](int p, int l) {
      return p < n && l <= hs[p].depth_o - 2 ? hs[p].path_o[l] - T.pw_base : -1;
    });
  for (int p = 0; p < n; ++p) {
    Tables tb;
    alloc_tables(phases + size_t(p) * per, T, tb);
    build_tables(T, hs[p].xo, 1.0, hs[p].Xo, hs[p].depth_o - 2, tb, tid, BG_T);
  }
  batch_sources<GRP>(T, srcs, [&](int p, int& leaf, int& l, const int*& Xl) {
    l = p < n ? hs[p].depth_o - 1 : -1;
    if (l < 0) return;
    leaf = hs[p].path_o[l];
    Xl = hs[p].Xo[l];
  });
  for (int i = tid; i < GRP * 4 * BG_W; i += BG_T) (&dsum[0][0][0])[i] = 0.0;
  __syncthreads();
  for (int l = 2; l <= top; ++l)
    for (int r = 0; r < rows.n[l]; ++r) {
      const double2* row = T.inc + size_t(rows.row[l][r]) * S::H;
      const int np = rows.npt[l][r];
      const unsigned char* pts = rows.pt[l][r];
      auto run = [&](auto nt) {
        constexpr int N = decltype(nt)::value;
        const double2* ex[N];
        const double2 *ey[N], *ez[N];
        double acc[N][3];
#pragma unroll
        for (int t = 0; t < N; ++t) {
          const int jb = 2 * t + (lane >> 4), jc = 2 * t + (q4 >> 1);
          auto lev = [&](int j, int ax) {
            return phases + size_t(pts[min(j, np - 1)]) * per + 3 * S::DW + (l - 2) * 3 * S::D + ax * S::D;
          };
          ex[t] = jb < np ? lev(jb, 0) : nullptr;
          ey[t] = lev(jc, 1);
          ez[t] = lev(jc, 2);
          acc[t][0] = acc[t][1] = acc[t][2] = 0.0;
        }
        row_products<NP, N, 4>(T, row, tab, ex, [&](int t, int iz, int iy, double2 sv) {
          const double2 u = cmul(cmul(ez[t][iz], ey[t][iy]), sv);
          if (q4 & 1) {
            acc[t][0] += u.y;  // x derivative
          } else {
            acc[t][0] += u.x;
            acc[t][1] += u.y * double(iy - ND);
            acc[t][2] += u.y * double(iz - ND);
          }
        });
#pragma unroll
        for (int t = 0; t < N; ++t) {
#pragma unroll
          for (int k = 0; k < 3; ++k)
            for (int o = 4; o < 32; o <<= 1) acc[t][k] += __shfl_xor_sync(0xffffffffu, acc[t][k], o);
          const int j = 2 * t + (lane >> 1);
          if (lane < 4 && j < np) {
            const int p = pts[j];
            const double c = c_level[l], dk = c * level_dk(T, l);
            if (lane & 1) {
              dsum[p][1][warp] += dk * acc[t][0];
            } else {
              dsum[p][0][warp] += c * acc[t][0];
              dsum[p][2][warp] += dk * acc[t][1];
              dsum[p][3][warp] += dk * acc[t][2];
            }
          }
        }
        __syncwarp();
      };
      if (NT > 1 && np > 2) run(std::integral_constant<int, NT>{});
      else run(std::integral_constant<int, 1>{});
    }
  // the k = 0 mode is left out, as in Ewald summation: a neutral system has
  // g(0) = 0, but all particles but one carry the net charge -q, whose
  // k = 0 term is the uniform neutralising background's business
  const int k_zero = (NW * S::DW + NW) * S::DW + NW;
  const double dk0 = T.delta_k[0];
  const int pool_n = 0;  // arrivals in the overflow pool are folded into the slots before this kernel runs
  for (int g = 0; g < n; ++g) {
    const Header& h = hs[g];
    const double q = h.q;
    Tables uu;
    alloc_tables(phases + size_t(g) * per, T, uu);
    double v[4] = {0, 0, 0, 0};  // phi and its gradient, window
    for (int k = tid; k < S::HW; k += BG_T) {
      if (k == k_zero) continue;
      const double2 u = phase_at(uu.root, k, S::DW);
      const double2 gk = T.out_root[k];
      const double bx = gk.x - q * u.x, by = gk.y - q * u.y;
      const double w = T.W[k];
      v[0] += (u.x * bx + u.y * by) * w;
      const double im = (u.y * bx - u.x * by) * w;  // Im(u conj(b))
      const int ix = k % S::DW, iy = (k / S::DW) % S::DW, iz = k / (S::DW * S::DW);
      v[1] += dk0 * (ix - NW) * im;
      v[2] += dk0 * (iy - NW) * im;
      v[3] += dk0 * (iz - NW) * im;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) v[a] *= c_window;
    const double b = level_box(T, h.depth_o - 1);
    batch_near<GRP>(T, srcs, g, h.xo, b, pool_n, [&](double qj, double dx, double dy, double dz, double r2) {
      const double r = sqrt(r2);
      v[0] += qj * poly(r, b);
      const double gr = qj * poly.deriv(r, b) / r;
      v[1] += gr * dx;
      v[2] += gr * dy;
      v[3] += gr * dz;
    });
    batch_block_sum<4>(v, red);
    if (tid == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
        for (int w = 0; w < BG_W; ++w) v[a] += dsum[g][a][w];
      double cself = 0.5 * c_window * sum_w - self_w;
      for (int l = 2; l <= h.depth_o - 2; ++l) {
        v[0] -= c_level[l] * q * sum_d2;
        cself += 0.5 * c_level[l] * sum_d2 - Sl[l];
      }
      int c = 0;
#pragma unroll
      for (int k = 0; k < GRP; ++k)
        if (k == g) c = cand[k];
      phi_out[c] = v[0] + 2.0 * q * cself;
      if (field_out)
        for (int a = 0; a < 3; ++a) field_out[3 * size_t(c) + a] = -v[1 + a];
    }
  }
}

using PotentialKernel = void (*)(DevTree, const int*, const int*, int, double, double, double, double, const double*,
                                 double*, double*);
PotentialKernel potential_kernel(int np, int grp) {
  switch (np) {
    case 7: return k_potential_batch<7, 1>;
    case 13: return grp > 1 ? k_potential_batch<13, BG_GROUP> : k_potential_batch<13, 1>;
    case 19: return grp > 1 ? k_potential_batch<19, BG_GROUP> : k_potential_batch<19, 1>;
    case 25: return grp > 1 ? k_potential_batch<25, BG_GROUP> : k_potential_batch<25, 1>;
    default: throw std::invalid_argument("unsupported residual polynomial");
  }
}

// the shift kernel for a residual polynomial of np coefficients (3, 6, 9, 12 digits)
using ShiftKernel = void (*)(DevTree, ShiftArgs, const OneMove);
ShiftKernel shift_kernel(int np) {
  switch (np) {
    case 7: return k_shift<7>;
    case 13: return k_shift<13>;
    case 19: return k_shift<19>;
    case 25: return k_shift<25>;
    default: throw std::invalid_argument("unsupported residual polynomial");
  }
}

size_t tables_smem(const DevTree& T, int lmax, int copies) {
  size_t per = 3 * size_t(2 * T.n_window + 1) + size_t(std::max(lmax - 1, 0)) * 3 * (2 * T.n_diff + 1);
  return per * copies * sizeof(double2);
}

}  // namespace

// ---------------------------------------------------------------------------
void DmkTree::launch_shift(const int* d_idx, const double* d_disp, const double* d_u, double beta, int move, int mode,
                           double* d_dE, int* d_acc, long one_i, const double* one_d) {
  DevTree& D = dev_;
  const double pi = 3.14159265358979323846;
  OneMove one{int(one_i), {0, 0, 0}};
  if (one_d) std::copy(one_d, one_d + 3, one.d);
  ShiftArgs a{};
  a.idx = d_idx;
  a.disp = d_disp;
  a.u = d_u;
  a.beta = beta;
  a.move = move;
  a.mode = mode;
  a.dE_out = d_dE;
  a.acc_out = d_acc;
  a.c_window = std::pow(D.delta_k[0], 3) / std::pow(2 * pi, 3);
  a.partials = D.partials;
  a.counter = D.counter;
  a.prop = D.prop;
  ensure_move_resources();
  a.cur = use_cursor_ ? d_cursor_ : nullptr;
  a.ptab = ptab_;
  a.ptab_per = ptab_per_;
  a.host_out = one_d ? slot_dev_ : nullptr;
  size_t smem = tables_smem(D, D.max_depth, 2);
  time_begin(0);
  shift_kernel(D.n_poly)<<<unsigned(shift_grid_), SH_T, smem, st_>>>(D, a, one);
  PDMK_LAUNCH_CHECK();
  time_end(0);
}

void DmkTree::launch_shift_cursor(int move) {
  // proposals, outputs, mode and beta come from *d_cursor_ at run time
  use_cursor_ = true;
  launch_shift(nullptr, nullptr, nullptr, 0.0, move, 1, nullptr, nullptr);
  use_cursor_ = false;
}

// Per-tree resources of the move kernels, set up before any graph capture
// (no allocation or attribute change may happen inside a capture).
void DmkTree::ensure_move_resources() {
  DevTree& D = dev_;
  if (!ptab_) {
    ptab_per_ = 3L * (2 * D.n_window + 1) + long(MAX_LEVELS + 1) * 3 * (2 * D.n_diff + 1);
    ptab_ = static_cast<double2*>(alloc(sizeof(double2) * 2 * size_t(ptab_per_)));
    d_cursor_ = static_cast<MoveCursor*>(alloc(sizeof(MoveCursor)));
  }
  ensure_shift_config();
  ensure_rows(true, true);
}

// Grid size and dynamic shared memory limit of the shift kernel (no allocation).
void DmkTree::ensure_shift_config() {
  DevTree& D = dev_;
  if (shift_grid_ == 0) {
    int dev = 0, sms = 148;
    PDMK_CUDA(cudaGetDevice(&dev));
    PDMK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    shift_grid_ = 3 + sms;
    const size_t smem = tables_smem(D, D.max_depth, 2);
    raise_smem_limit(reinterpret_cast<const void*>(shift_kernel(D.n_poly)), smem);
  }
}

// Capture kGraphMoves sequential moves (shift, update, commit) into one
// executable graph; with timed != 0 external event records bracket each
// update so its duration can be read after the graph ran.
void DmkTree::build_mc_graph(int timed) {
  ensure_move_resources();
  if (timed && graph_ev_.empty()) {
    graph_ev_.resize(2 * kGraphMoves);
    for (auto& e : graph_ev_) PDMK_CUDA(cudaEventCreate(&e));
  }
  cudaGraph_t g;
  const long long launches0 = g_launch_count.load();  // captured launches do not run here
  capturing_ = true;
  PDMK_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
  try {
    for (int b = 0; b < kGraphMoves; ++b) {
      launch_shift_cursor(b);
      if (timed) PDMK_CUDA(cudaEventRecordWithFlags(graph_ev_[2 * b], st_, cudaEventRecordExternal));
      launch_update();
      if (timed) PDMK_CUDA(cudaEventRecordWithFlags(graph_ev_[2 * b + 1], st_, cudaEventRecordExternal));
    }
  } catch (...) {
    capturing_ = false;
    cudaStreamEndCapture(st_, &g);
    throw;
  }
  PDMK_CUDA(cudaStreamEndCapture(st_, &g));
  capturing_ = false;
  g_launch_count.store(launches0);
  PDMK_CUDA(cudaGraphInstantiate(&mc_graph_[timed], g, 0));
  PDMK_CUDA(cudaGraphDestroy(g));
}

void DmkTree::launch_update(bool force) {
  DevTree& D = dev_;
  // rows: root, up to 2 x 28 receivers per expansion level, commit
  // x: one mode per thread; y: receiver ranges, enough for ~16 warps per SM
  const int gx = (std::max(D.H, D.Hw) + UPD_T - 1) / UPD_T;
  const int gy = std::max(1, std::min(8, (16 * (shift_grid_ - 3) * 32 / UPD_T + gx - 1) / std::max(gx, 1)));
  const dim3 grid{unsigned(gx), unsigned(gy), 1u};
  time_begin(1);
  k_update<<<grid, UPD_T, 0, st_>>>(D, ptab_, ptab_per_, force,
                                      force && slot_ ? reinterpret_cast<int*>(slot_dev_ + 6) : nullptr);
  PDMK_LAUNCH_CHECK();
  time_end(1);
}


cudaEvent_t DmkTree::take_event() {
  if (!ev_pool_.empty()) {
    cudaEvent_t e = ev_pool_.back();
    ev_pool_.pop_back();
    return e;
  }
  cudaEvent_t e;
  PDMK_CUDA(cudaEventCreate(&e));
  return e;
}

void DmkTree::time_begin(int cls) {
  if (!timing_ || capturing_) return;
  ev_cur_[cls] = take_event();
  PDMK_CUDA(cudaEventRecord(ev_cur_[cls], st_));
}

void DmkTree::time_end(int cls) {
  if (!timing_ || capturing_ || !ev_cur_[cls]) return;
  cudaEvent_t e = take_event();
  PDMK_CUDA(cudaEventRecord(e, st_));
  ev_open_.push_back({cls, {ev_cur_[cls], e}});
  ev_cur_[cls] = nullptr;
}

void DmkTree::get_timing(double* out, bool reset) {
  PDMK_CUDA(cudaStreamSynchronize(st_));
  for (auto& o : ev_open_) {
    float ms = 0;
    PDMK_CUDA(cudaEventElapsedTime(&ms, o.second.first, o.second.second));
    t_ms_[o.first] += ms;
    t_cnt_[o.first] += 1;
    ev_pool_.push_back(o.second.first);
    ev_pool_.push_back(o.second.second);
  }
  ev_open_.clear();
  for (int c = 0; c < 4; ++c) {
    out[2 * c] = t_ms_[c];
    out[2 * c + 1] = double(t_cnt_[c]);
    if (reset) {
      t_ms_[c] = 0;
      t_cnt_[c] = 0;
    }
  }
}

void DmkTree::get_work(double* out) {
  unsigned long long w[3];
  PDMK_CUDA(cudaMemcpyAsync(w, dev_.work, sizeof(w), cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
  for (int c = 0; c < 3; ++c) out[c] = double(w[c]);
}

void DmkTree::reset_work() { PDMK_CUDA(cudaMemsetAsync(dev_.work, 0, 3 * sizeof(unsigned long long), st_)); }

double DmkTree::eval_shift_energy(long i, double dx, double dy, double dz, double* parts) {
  double disp[3] = {dx, dy, dz};
  // the proposal goes with the launch and the result comes through mapped
  // memory: the copies took 3 and 5 us of a trial's 46
  if (!slot_tried_) {
    slot_ = take_host_slot(&slot_dev_);
    slot_tried_ = true;
  }
  launch_shift(nullptr, nullptr, nullptr, 0.0, 0, 0, nullptr, nullptr, i, disp);
  double got[6];
  if (slot_) {
    PDMK_CUDA(cudaStreamSynchronize(st_));
    std::copy(slot_, slot_ + 6, got);
  } else {
    Proposal P;
    PDMK_CUDA(cudaMemcpyAsync(&P, dev_.prop, sizeof(Proposal), cudaMemcpyDeviceToHost, st_));
    PDMK_CUDA(cudaStreamSynchronize(st_));
    got[0] = P.dE;
    std::copy(P.parts, P.parts + 5, got + 1);
  }
  if (parts) std::copy(got + 1, got + 6, parts);
  last_i_ = i;
  last_d_[0] = dx;
  last_d_[1] = dy;
  last_d_[2] = dz;
  last_valid_ = true;
  return got[0];
}

int DmkTree::update_shift(long i, double dx, double dy, double dz) {
  // the reference requires the same arguments as the preceding
  // eval_shift_energy (src/tree.cpp:471-489); recompute when they differ
  if (!(last_valid_ && last_i_ == i && last_d_[0] == dx && last_d_[1] == dy && last_d_[2] == dz))
    eval_shift_energy(i, dx, dy, dz, nullptr);
  launch_update(true);
  last_valid_ = false;
  diff_cached_ = false;
  mark_moved();
  if (!slot_) return check_device_error();
  PDMK_CUDA(cudaStreamSynchronize(st_));
  return *reinterpret_cast<const volatile int*>(slot_ + 6);
}

// The deferred-update list of a tree, its marks and the folded difference
// table, kept with the tree for its later sequences.
void DmkTree::ensure_pending(int cap) {
  DevTree& D = dev_;
  if (!d_oct_) {
    int stride = 0, n_oct = 0;
    switch (D.n_poly) {
      case 7: stride = ModesOf<7>::STR, n_oct = ModesOf<7>::OCT; break;
      case 13: stride = ModesOf<13>::STR, n_oct = ModesOf<13>::OCT; break;
      case 19: stride = ModesOf<19>::STR, n_oct = ModesOf<19>::OCT; break;
      case 25: stride = ModesOf<25>::STR, n_oct = ModesOf<25>::OCT; break;
      default: throw std::invalid_argument("unsupported residual polynomial");
    }
    const int n_pw = D.level_start[D.pw_hi + 1] - D.pw_base;
    d_oct_ = static_cast<double*>(alloc(sizeof(double) * size_t(n_oct)));
    k_fold_d2<<<unsigned((n_oct + 255) / 256), 256, 0, st_>>>(D, stride, n_oct, d_oct_);
    PDMK_LAUNCH_CHECK();
    d_touched_ = static_cast<int*>(alloc(sizeof(int) * (size_t(n_pw) + 1)));
    d_n_list_ = d_touched_ + n_pw;
  }
  if (cap > pending_cap_) {
    d_pending_ = alloc(sizeof(Pending) * size_t(cap));
    pending_cap_ = cap;
  }
}

// Empties the list, before a sequence that fills it.
void DmkTree::clear_pending() {
  const int n_pw = dev_.level_start[dev_.pw_hi + 1] - dev_.pw_base;
  PDMK_CUDA(cudaMemsetAsync(d_touched_, 0, sizeof(int) * (size_t(n_pw) + 1), st_));
}

// Brings the expansion rows up to date with the listed moves.
void DmkTree::flush_pending() {
  launch_flush_outgoing(dev_, static_cast<const Pending*>(d_pending_), d_n_list_, d_touched_, st_);
  launch_incoming_touched(d_touched_);
}

// One cooperative launch per kMcChunk moves on every SM (k_mc). The grid is
// the SM count, which the occupancy query confirms can be co-resident; the
// cooperative launch refuses to start otherwise, so the grid barriers inside
// cannot wait on a block that never runs.
void DmkTree::mc_run_persistent(int n_moves, const int* d_idx, const double* d_disp, const double* d_u, double beta,
                                double* d_dE, int* d_acc) {
  DevTree& D = dev_;
  ensure_rows(true, true);
  const size_t smem = tables_smem(D, D.max_depth, 2);
  const McKernel kern = mc_kernel(D.n_poly);
  if (mc_grid_ == 0) {
    int dev = 0, sms = 0, coop = 0;
    PDMK_CUDA(cudaGetDevice(&dev));
    PDMK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PDMK_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) throw CudaError("device does not support cooperative launches");
    raise_smem_limit(reinterpret_cast<const void*>(kern), smem);
    int per_sm = 0;
    PDMK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, MC_T, smem));
    if (per_sm < 1) throw CudaError("persistent Metropolis kernel does not fit on one SM");
    mc_partials_ = static_cast<double*>(alloc(sizeof(double) * 8 * size_t(sms)));
    mc_sync_ = static_cast<unsigned int*>(alloc(64));
    mc_grid_ = sms;
  }
  if (mc_run_long(n_moves, d_idx, d_disp, d_u, beta, d_dE, d_acc)) return;
  const double pi = 3.14159265358979323846;
  for (int m0 = 0; m0 < n_moves; m0 += kMcChunk) {
    const int cnt = std::min(kMcChunk, n_moves - m0);
    PDMK_CUDA(cudaMemsetAsync(mc_sync_, 0, 64, st_));
    McArgs a{};
    a.idx = d_idx + m0;
    a.disp = d_disp + 3 * size_t(m0);
    a.u = d_u + m0;
    a.beta = beta;
    a.n_moves = cnt;
    a.dE_out = d_dE ? d_dE + m0 : nullptr;
    a.acc_out = d_acc ? d_acc + m0 : nullptr;
    a.c_window = std::pow(D.delta_k[0], 3) / std::pow(2 * pi, 3);
    a.partials = mc_partials_;
    a.arrivals = mc_sync_;
    a.spin_limit = 1LL << 21;  // about a second of polling
    void* args[] = {&D, &a};
    time_begin(2);
    PDMK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(unsigned(mc_grid_)),
                                          dim3(unsigned(MC_T)), args, smem, st_));
    PDMK_LAUNCH_CHECK();
    time_end(2);
  }
}

// The same for a sequence long enough to defer its row updates (k_mc_long);
// false when it is not. The passes that bring the rows up to date cost with the
// rows' bytes, an update move by move with the number of moves. Both forms take
// the same time at (moves of up to 0.3 spacings per axis at beta = 1; digits, rows,
// MB of rows): fewer than 8 moves up to 31 MB and for 3 digits up to 146 MB;
// 14 (6, 576, 75); 23 (9, 576, 280); 48 (6, 4672, 607); 38 (12, 576, 699); 74 (9,
// 4672, 2274); 106 (9, 7776, 3785); above 128 (12, 7632, 9261). The line lies along
// these. Deferred / move by move, us a call: 24 moves at 280 MB 498 / 505, 128 at
// 280 MB 1406 / 2518, 32 at 699 MB 1041 / 964, 128 at 2274 MB 2583 / 3647.
bool DmkTree::mc_run_long(int n_moves, const int* d_idx, const double* d_disp, const double* d_u, double beta, double* d_dE,
                          int* d_acc) {
  DevTree& D = dev_;
  const int n_pw = D.pw_hi >= D.pw_lo ? D.level_start[D.pw_hi + 1] - D.pw_base : 0;
  const long mb = 16L * n_pw * D.H / 1000000;
  if (!inc_formed_ || n_pw == 0 || n_moves < 8 + std::min(mb, 650L) / 16 + std::max(mb - 650, 0L) / 52) return false;
  // A longer list makes each move's pair sums longer (5 ns per listed move at
  // N = 1e5, 7.4 ns at 1e6), a shorter one updates the rows more often (0.38 and
  // 2.1 ms). 2000 moves at N = 1e5 / 4000 at 1e6 (9 digits, positions
  // read at the end): 20.8 / 75.1 ms at 384 moves a list, 20.7 / 71.3 at 512, 20.9 /
  // 69.8 at 768, 21.3 / 68.1 at 1024, 23.6 / 69.9 at 2048.
  const int longest = n_pw >= 1024 ? 1024 : 512;
  // What this form keeps is allocated and filled by its first call outside a
  // capture: memory taken inside one belongs to the graph. Until then a captured
  // sequence runs move by move.
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  PDMK_CUDA(cudaStreamIsCapturing(st_, &cs));
  if (cs != cudaStreamCaptureStatusNone &&
      !(mcl_grid_ > 0 && box_lists_ready_ && d_oct_ && pending_cap_ >= std::min(longest, kPendPerBlock * mcl_grid_)))
    return false;
  const McLongKernel kern = mc_long_kernel(D.n_poly);
  const size_t smem = tables_smem(D, D.max_depth, 4) + mc_long_smem(D.n_poly, kPendPerBlock);
  if (mcl_grid_ == 0) {
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    PDMK_CUDA(cudaGetDevice(&dev));
    PDMK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PDMK_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) throw CudaError("device does not support cooperative launches");
    raise_smem_limit(reinterpret_cast<const void*>(kern), smem);
    PDMK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, MCL_T, smem));
    // a thread holds at most two of its block's modes
    if (per_sm < 1 || sms < 144) return false;
    d_pos4_ = alloc(sizeof(double4) * size_t(N_));
    d_packets_ = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * 4 * size_t(sms) + 64));
    mcl_grid_ = sms;
  }
  prepare_box_lists();
  const int chunk = std::min(longest, kPendPerBlock * mcl_grid_);
  ensure_pending(chunk);
  const double pi = 3.14159265358979323846;
  for (int m0 = 0; m0 < n_moves; m0 += chunk) {
    const int cnt = std::min(chunk, n_moves - m0);
    McLongArgs a{};
    a.idx = d_idx + m0;
    a.disp = d_disp + 3 * size_t(m0);
    a.u = d_u + m0;
    a.beta = beta;
    a.n_moves = cnt;
    a.dE_out = d_dE ? d_dE + m0 : nullptr;
    a.acc_out = d_acc ? d_acc + m0 : nullptr;
    a.c_window = std::pow(D.delta_k[0], 3) / std::pow(2 * pi, 3);
    a.packets = d_packets_;
    a.committed = reinterpret_cast<unsigned int*>(d_packets_ + 4 * size_t(mcl_grid_));
    a.pos4 = static_cast<double4*>(d_pos4_);
    a.spin_limit = 1LL << 21;  // about a second of polling
    a.list = static_cast<Pending*>(d_pending_);
    a.n_list = d_n_list_;
    a.touched = d_touched_;
    a.oct = d_oct_;
    a.per_block = kPendPerBlock;
    clear_pending();
    PDMK_CUDA(cudaMemsetAsync(d_packets_, 0, sizeof(unsigned long long) * 4 * size_t(mcl_grid_) + 64, st_));
    k_gather_moves<<<unsigned((cnt + 255) / 256), 256, 0, st_>>>(D, a.idx, cnt, a.pos4);
    PDMK_LAUNCH_CHECK();
    void* args[] = {&D, &a};
    time_begin(2);
    PDMK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(unsigned(mcl_grid_)),
                                          dim3(unsigned(MCL_T)), args, smem, st_));
    PDMK_LAUNCH_CHECK();
    flush_pending();
    time_end(2);
  }
  return true;
}

void DmkTree::mc_run_device(int n_moves, const int* d_idx, const double* d_disp, const double* d_u, double beta,
                            double* d_dE, int* d_acc) {
  if (mc_mode_ == 0) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    PDMK_CUDA(cudaStreamIsCapturing(st_, &cs));
    captured_moves_ = captured_moves_ || cs != cudaStreamCaptureStatusNone;
    if (n_moves > 0) mc_run_persistent(n_moves, d_idx, d_disp, d_u, beta, d_dE, d_acc);
    last_valid_ = false;
    diff_cached_ = false;
    mark_moved();
    return;
  }
  ensure_move_resources();
  int m = 0;
  // whole batches run as one captured graph each; with timing on, one batch
  // in kTimedEvery runs the graph variant whose updates are bracketed by
  // event records (those records slow the graph, so only a sample carries them)
  while (n_moves - m >= kGraphMoves) {
    const int timed = (timing_ && (timed_batches_++ % kTimedEvery) == 0) ? 1 : 0;
    if (!mc_graph_[timed]) build_mc_graph(timed);
    MoveCursor c{d_idx, d_disp, d_u, d_dE, d_acc, m, 1, beta};
    PDMK_CUDA(cudaMemcpyAsync(d_cursor_, &c, sizeof(c), cudaMemcpyHostToDevice, st_));
    PDMK_CUDA(cudaGraphLaunch(mc_graph_[timed], st_));
    g_launch_count.fetch_add(2 * kGraphMoves, std::memory_order_relaxed);  // shift + update per move
    if (timed) {
      // the events are reused by the next launch: read them now
      PDMK_CUDA(cudaStreamSynchronize(st_));
      for (int b = 0; b < kGraphMoves; ++b) {
        float ms = 0;
        PDMK_CUDA(cudaEventElapsedTime(&ms, graph_ev_[2 * b], graph_ev_[2 * b + 1]));
        t_ms_[1] += ms;
        t_cnt_[1] += 1;
      }
    }
    m += kGraphMoves;
  }
  for (; m < n_moves; ++m) {
    launch_shift(d_idx, d_disp, d_u, beta, m, 1, d_dE, d_acc);
    launch_update();
  }
  last_valid_ = false;
  diff_cached_ = false;
  mark_moved();
}

// The batch kernels' groups: BG_GROUP particles a block in Morton order where that
// pays (in_pairs; order: room for m indices, or null), else one.
int DmkTree::batch_groups(int m, const int* d_idx, int* order) {
  const int grp = order && in_pairs(dev_.n_poly, m) ? BG_GROUP : 1;
  if (grp > 1) {
    k_order_particles<<<1, 1024, 0, st_>>>(dev_, d_idx, m, order);
    PDMK_LAUNCH_CHECK();
  }
  return grp;
}

// The tree's own index array for the order; null under capture: a graph may be
// replayed on a stream beside the tree's, where a direct call would share it (a
// captured batch runs one candidate a block: 1.30 instead of 1.04 ms for 4096 at N
// = 1e6, 9 digits).
int* DmkTree::batch_order(int m) {
  if (!in_pairs(dev_.n_poly, m)) return nullptr;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  PDMK_CUDA(cudaStreamIsCapturing(st_, &cs));
  if (cs != cudaStreamCaptureStatusNone) return nullptr;
  if (m > order_cap_) {
    order_cap_ = std::max(m, 2 * order_cap_);
    d_order_ = static_cast<int*>(alloc(sizeof(int) * size_t(order_cap_)));
  }
  return d_order_;
}

void DmkTree::launch_shift_batch(int m, const int* d_idx, const double* d_disp, int* order, double* d_dE) {
  DevTree& D = dev_;
  ensure_rows(true, true);
  const int grp = batch_groups(m, d_idx, order);
  const size_t smem = batch_smem(D.n_poly, D.max_depth, 2 * grp);
  const ShiftBatchKernel kern = shift_batch_kernel(D.n_poly, grp);
  raise_smem_limit(reinterpret_cast<const void*>(kern), smem);
  const double pi = 3.14159265358979323846;
  const double c_window = std::pow(D.delta_k[0], 3) / std::pow(2 * pi, 3);
  kern<<<unsigned((m + grp - 1) / grp), BG_T, smem, st_>>>(D, d_idx, d_disp, grp > 1 ? order : nullptr, m, c_window, sum_d2_,
                                                           d_dE);
  PDMK_LAUNCH_CHECK();
}

// All candidates in one launch of k_shift_batch.
void DmkTree::shift_batch_device(int m, const int* d_idx, const double* d_disp, double* d_dE) {
  if (m <= 0) return;
  launch_shift_batch(m, d_idx, d_disp, batch_order(m), d_dE);
  last_valid_ = false;
}

// ---------------------------------------------------------------------------
// Candidate batch through a fixed static device buffer. For callers that may
// not allocate device memory once the tree exists (a process that budgets its
// device memory up front, a host thread that must not enter the allocator
// between steps): the candidates' indices and displacements are staged into
// g_static_scratch and their energy shifts come back through it, and the
// batch is the same launch of k_shift_batch as the allocating batch (its phase
// tables live in shared memory; the order of a large batch in the array). The
// array's device address is looked up once per device, with that device
// current. Nothing in the buffer has to start at zero: every call writes the
// inputs it reads, and the kernel writes every output before it is read.
// Calls that overlap in time on one device (two host threads, two trees on
// different streams) share the buffer and race; serialise them.
namespace {
constexpr int kStaticMaxMoves = 4096;  // candidates per call
constexpr size_t kOffIdx = 0;
constexpr size_t kOffDisp = kOffIdx + sizeof(int) * kStaticMaxMoves;
constexpr size_t kOffDE = kOffDisp + sizeof(double) * 3 * kStaticMaxMoves;
constexpr size_t kOffOrder = kOffDE + sizeof(double) * kStaticMaxMoves;
constexpr size_t kStaticBytes = kOffOrder + sizeof(int) * kStaticMaxMoves;  // 160 KB

static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

unsigned char* static_scratch() {
  static std::mutex mu;
  static void* addr[64] = {};
  int dev = 0;
  PDMK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) throw std::runtime_error("device ordinal out of range for the static scratch table");
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || !p)
      throw CudaError(std::string("cudaGetSymbolAddress(static shift scratch): ") + cudaGetErrorString(e));
    addr[dev] = p;
  }
  return static_cast<unsigned char*>(addr[dev]);
}
}  // namespace

void DmkTree::shift_batch_static(int m, const long* h_idx, const double* h_disp, double* h_dE) {
  DevTree& D = dev_;
  if (m < 0 || m > kStaticMaxMoves)
    throw std::invalid_argument("static scratch holds at most " + std::to_string(kStaticMaxMoves) +
                                " candidates per call, got " + std::to_string(m));
  if (m == 0) return;
  unsigned char* base = static_scratch();
  int* s_idx = reinterpret_cast<int*>(base + kOffIdx);
  double* s_disp = reinterpret_cast<double*>(base + kOffDisp);
  double* s_dE = reinterpret_cast<double*>(base + kOffDE);
  // indices narrowed through a stack buffer (pageable copies are staged
  // before cudaMemcpyAsync returns, so the buffer may be reused at once)
  int chunk[512];
  for (int c0 = 0; c0 < m; c0 += 512) {
    const int nc = std::min(512, m - c0);
    for (int c = 0; c < nc; ++c) chunk[c] = int(h_idx[c0 + c]);
    PDMK_CUDA(cudaMemcpyAsync(s_idx + c0, chunk, sizeof(int) * nc, cudaMemcpyHostToDevice, st_));
  }
  PDMK_CUDA(cudaMemcpyAsync(s_disp, h_disp, sizeof(double) * 3 * m, cudaMemcpyHostToDevice, st_));
  // both forms of the kernel are loaded by the first call, so that no later
  // one enters the driver's allocator
  for (int grp : {1, BG_GROUP})
    raise_smem_limit(reinterpret_cast<const void*>(shift_batch_kernel(D.n_poly, grp)),
                     batch_smem(D.n_poly, D.max_depth, 2 * grp));
  cudaFuncAttributes fa;
  PDMK_CUDA(cudaFuncGetAttributes(&fa, k_order_particles));
  launch_shift_batch(m, s_idx, s_disp, reinterpret_cast<int*>(base + kOffOrder), s_dE);
  PDMK_CUDA(cudaMemcpyAsync(h_dE, s_dE, sizeof(double) * m, cudaMemcpyDeviceToHost, st_));
  PDMK_CUDA(cudaStreamSynchronize(st_));
}

// Metropolis sequences of many trees (k_mc_rep), ordered after all their streams'
// earlier work on the first tree's stream; d_err[i]: the trees' error words after
// it, for the host to read with the results. Four launches per REP_CHUNK moves
// serve the whole set (a clear, the moves, the outgoing and the incoming rows):
// with a clear and two row launches for each tree, and its error word read by
// itself, sets of many small trees paid more for these than for a short
// sequence's moves.
void DmkTree::replicas_mc_run(const std::vector<DmkTree*>& ts, int m, const int* d_idx, const double* d_disp,
                              const double* d_u, double beta, double* d_dE, int* d_acc, int* d_err) {
  if (ts.empty() || m <= 0) return;
  const size_t nt = ts.size();
  const int np = ts[0]->dev_.n_poly;
  size_t smem = 0;
  bool deferred = nt > 1;  // one tree has every SM to itself
  for (DmkTree* t : ts) {
    if (t->dev_.n_poly != np) throw std::invalid_argument("replicas must share the digits setting");
    t->ensure_packed();
    t->ensure_rows(true, true);
    smem = std::max(smem, tables_smem(t->dev_, t->dev_.max_depth, 2));
    deferred = deferred && (t->inc_formed_ || t->dev_.pw_hi < t->dev_.pw_lo);
  }
  const int chunk = std::min(m, REP_CHUNK);
  std::vector<DevTree> trees(nt);
  std::vector<SequenceRows> rows(nt);
  int flush = 0, cubes = 0, inc = 0, n_pw_max = 0;
  if (deferred) {
    for (DmkTree* t : ts) {
      t->ensure_pending(chunk);
      if (t->dev_.pw_hi >= t->dev_.pw_lo) t->prepare_box_lists();
      cubes += t->n_cubes_;
    }
    for (size_t i = 0; i < nt; ++i) {
      DmkTree* t = ts[i];
      const DevTree& D = t->dev_;
      SequenceRows& r = rows[i];
      r.list = static_cast<Pending*>(t->d_pending_);
      r.n_list = t->d_n_list_;
      r.touched = t->d_touched_;
      r.oct = t->d_oct_;
      r.n_pw = D.pw_hi >= D.pw_lo ? D.level_start[D.pw_hi + 1] - D.pw_base : 0;
      r.cubes = t->d_cubes_;
      r.n_cubes = r.n_pw > 0 ? t->n_cubes_ : 0;
      // about 2^15 blocks for the set: more would pay their set-up for a few tiles
      r.slots = std::min(t->inc_slots(), std::max(1, (1 << 15) / std::max(cubes, 1)));
      flush = std::max(flush, flush_blocks(D));
      inc = std::max(inc, r.slots * r.n_cubes);
      n_pw_max = std::max(n_pw_max, r.n_pw);
      trees[i] = D;
    }
  }
  cudaStream_t st = ts[0]->st_;
  std::vector<cudaEvent_t> evs(nt);
  for (auto& e : evs) PDMK_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  if (deferred) {
    for (size_t i = 1; i < nt; ++i) {
      PDMK_CUDA(cudaEventRecord(evs[i], ts[i]->st_));
      PDMK_CUDA(cudaStreamWaitEvent(st, evs[i], 0));
    }
    unsigned char* d_set = nullptr;
    const size_t rows_at = (nt * sizeof(DevTree) + 15) & ~size_t(15);
    PDMK_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&d_set), rows_at + nt * sizeof(SequenceRows), st));
    const DevTree* d_trees = reinterpret_cast<const DevTree*>(d_set);
    const SequenceRows* d_rows = reinterpret_cast<const SequenceRows*>(d_set + rows_at);
    PDMK_CUDA(cudaMemcpyAsync(d_set, trees.data(), nt * sizeof(DevTree), cudaMemcpyHostToDevice, st));
    PDMK_CUDA(cudaMemcpyAsync(d_set + rows_at, rows.data(), nt * sizeof(SequenceRows), cudaMemcpyHostToDevice, st));
    const McRepKernel kern = mc_rep_kernel(np);
    smem += rep_lazy_smem(np);
    raise_smem_limit(reinterpret_cast<const void*>(kern), smem);
    RepArgs a{};
    a.trees = d_trees;
    a.m = m;
    a.idx = d_idx;
    a.disp = d_disp;
    a.u = d_u;
    a.beta = beta;
    a.dE_out = d_dE;
    a.acc_out = d_acc;
    a.rows = d_rows;
    const int n_diff = ts[0]->dev_.n_diff;
    for (a.m0 = 0; a.m0 < m; a.m0 += chunk) {
      a.cnt = std::min(chunk, m - a.m0);
      k_clear_set<<<set_grid(std::min(n_pw_max / 1024 + 1, 64), int(nt)), 256, 0, st>>>(d_rows, int(nt));
      PDMK_LAUNCH_CHECK();
      kern<<<unsigned(nt), REP_T, smem, st>>>(a);
      PDMK_LAUNCH_CHECK();
      launch_flush_set(n_diff, d_trees, d_rows, int(nt), flush, st);
      launch_incoming_set(n_diff, d_trees, d_rows, int(nt), inc, st);
    }
    k_errors_of_set<<<unsigned((nt + 127) / 128), 128, 0, st>>>(d_trees, int(nt), d_err);
    PDMK_LAUNCH_CHECK();
    PDMK_CUDA(cudaFreeAsync(d_set, st));
    PDMK_CUDA(cudaEventRecord(evs[0], st));
    for (size_t i = 1; i < nt; ++i) PDMK_CUDA(cudaStreamWaitEvent(ts[i]->st_, evs[0], 0));
  } else {
    // Deferred updates recompute incoming rows from the outgoing ones, which is
    // what accepted moves do to them only where a pass formed them so. A set
    // with a tree whose rows were not formed runs tree by tree.
    PDMK_CUDA(cudaEventRecord(evs[0], st));
    for (size_t i = 0; i < nt; ++i) {
      DmkTree* t = ts[i];
      if (i > 0) PDMK_CUDA(cudaStreamWaitEvent(t->st_, evs[0], 0));
      const size_t c = i * size_t(m);
      t->mc_run_persistent(m, d_idx + c, d_disp + 3 * c, d_u + c, beta, d_dE ? d_dE + c : nullptr,
                           d_acc ? d_acc + c : nullptr);
      PDMK_CUDA(cudaMemcpyAsync(d_err + i, t->dev_.err, sizeof(int), cudaMemcpyDeviceToDevice, t->st_));
      if (i > 0) {
        PDMK_CUDA(cudaEventRecord(evs[i], t->st_));
        PDMK_CUDA(cudaStreamWaitEvent(st, evs[i], 0));
      }
    }
  }
  for (auto& e : evs) PDMK_CUDA(cudaEventDestroy(e));  // released once the waits resolve
  for (DmkTree* t : ts) {
    t->last_valid_ = false;
    t->diff_cached_ = false;
    t->mark_moved();
  }
}

// Potentials and fields at many particles in one launch (k_potential_batch).
void DmkTree::potential_batch(int m, const int* d_idx, double* d_phi, double* d_field) {
  DevTree& D = dev_;
  if (m <= 0) return;
  ensure_packed();  // the near-field source lists read the slots only
  ensure_rows(true, true);
  int* order = batch_order(m);
  const int grp = batch_groups(m, d_idx, order);
  const size_t smem = batch_smem(D.n_poly, D.max_depth, grp);
  const PotentialKernel kern = potential_kernel(D.n_poly, grp);
  raise_smem_limit(reinterpret_cast<const void*>(kern), smem);
  const double pi = 3.14159265358979323846;
  const double c_window = std::pow(D.delta_k[0], 3) / std::pow(2 * pi, 3);
  const double self_w = ps_.psi0_0 / (2 * D.boxsize[2] * ps_.C0);
  kern<<<unsigned((m + grp - 1) / grp), BG_T, smem, st_>>>(D, d_idx, grp > 1 ? order : nullptr, m, c_window, self_w,
                                                           sum_w_, sum_d2_, d_Sl_, d_phi, d_field);
  PDMK_LAUNCH_CHECK();
}

}  // namespace pdmk
