// solver2d.cu -- the 2D Cauchy-kernel FMM of LibAran on the GPU, for a
// batch of independent systems solved in one pass (a forest).
//
// Reference: aran_solver2d_solve (aran/aransolver2d.c:1137-1204) driving
// aran_development2d_{p2m,m2m,m2l,l2l,local_evaluate}
// (aran/arandevelopment2d.c:167-346) over libvsg's quadtree, with the P2P
// kernel of tests/dummypot.c:62-76 (acc_i += q_j / (z_i - z_j)).
//
// Layout.  Particles are sorted by a 64-bit key (system id << 42 | 2x21-bit
// Morton code of the coordinates quantised in the system's box), so every
// system is one contiguous range and every quadtree node one sub-range.
// Nodes are level-major over the whole forest: level 0 holds one root per
// system.  Expansions are FP64 complex, p + 1 terms per node:
//   multipole  mult[k] = coefficient of z^{-k} (k = 1..p; k = 0 is the
//              constant term the reference keeps and never fills),
//   local      loc[k]  = coefficient of z^k (k = 0..p).
// The operators restate the reference's loops (aranlaurentseriesd.c:47-73,
// 358-452): M2M and L2L are Horner sums with Pascal-triangle binomials, M2L
// is the Laurent -> Taylor re-expansion, with one warp per node and one lane
// per output term.  The tree contract is the 3D one with 4 children: a node
// with more than maxbox points below the depth limit gets all 4 quadrants;
// same-depth non-adjacent children of adjacent nodes are far; adjacent
// leaves, and a leaf against all leaves below an adjacent internal node,
// are near.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "internal.cuh"
#include "f32x2.cuh"
#include "subdivide.cuh"

namespace aran {
namespace {

constexpr int kMaxOrder2d = 64;
constexpr int kSysShift = 42;   // 2 x 21 Morton bits below the system id

FMM_HD uint64_t spread2(uint64_t v) {
  v &= 0x1fffffull;
  v = (v | (v << 16)) & 0x0000ffff0000ffffull;
  v = (v | (v << 8)) & 0x00ff00ff00ff00ffull;
  v = (v | (v << 4)) & 0x0f0f0f0f0f0f0f0full;
  v = (v | (v << 2)) & 0x3333333333333333ull;
  v = (v | (v << 1)) & 0x5555555555555555ull;
  return v;
}

typedef cplx<double> zd;

__device__ __forceinline__ zd zmul(zd a, zd b) { return cmul(a, b); }
__device__ __forceinline__ zd zscale(zd a, double s) { return cmake(a.re * s, a.im * s); }
__device__ __forceinline__ zd zinv(zd a) {
  double r2 = a.re * a.re + a.im * a.im;
  double w = 1.0 / r2;
  return cmake(a.re * w, -a.im * w);
}
__device__ __forceinline__ double shfl_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------- keys/sort
// per system: lbx, lby, ubx, uby, scale x, scale y
// a non-finite coordinate or charge sets kErrNonFinite in *err, a point
// outside its system's closed box kErrOutside (its key is clamped into a
// boundary cell)
__global__ void k2_keys(int64_t n, int nsys, const int64_t *__restrict__ offs,
                        const double *__restrict__ sysbox, const double *__restrict__ xy,
                        const double *__restrict__ q, uint64_t *__restrict__ keys,
                        int *__restrict__ idx, int *__restrict__ err) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  // last system s with offs[s] <= i
  int lo = 0, hi = nsys;  // answer in [lo, hi)
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (offs[mid] <= i) lo = mid; else hi = mid;
  }
  const double *b = sysbox + 6 * lo;
  const double x = xy[2 * i], y = xy[2 * i + 1];
  if (!(isfinite(x) && isfinite(y) && isfinite(q[i]))) atomicOr(err, kErrNonFinite);
  const int64_t ix = cell_index(cell_pos(x, b[0], b[4])), iy = cell_index(cell_pos(y, b[1], b[5]));
  if (cell_outside(ix) || cell_outside(iy)) atomicOr(err, kErrOutside);
  uint64_t qx = (uint64_t)cell_clamp(ix);
  uint64_t qy = (uint64_t)cell_clamp(iy);
  keys[i] = ((uint64_t)lo << kSysShift) | spread2(qx) | (spread2(qy) << 1);
  idx[i] = (int)i;
}

__global__ void k2_gather(int64_t n, const int *__restrict__ perm, const double *__restrict__ xy,
                          const double *__restrict__ q, const uint64_t *__restrict__ keys,
                          const double *__restrict__ sysbox, double *__restrict__ sx,
                          double *__restrict__ sy, double *__restrict__ sq,
                          float4 *__restrict__ hl) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int o = perm[i];
  const double x = xy[2 * (int64_t)o], y = xy[2 * (int64_t)o + 1];
  sx[i] = x;
  sy[i] = y;
  sq[i] = q[o];
  if (hl) {              // FP32 hi + lo positions of the mixed near field, from the
                         // corner of the system's box
    const double *b = sysbox + 6 * (keys[i] >> kSysShift);
    const double bx = x - b[0], by = y - b[1];
    const float hx = (float)bx, hy = (float)by;
    hl[i] = make_float4(hx, hy, (float)(bx - (double)hx), (float)(by - (double)hy));
  }
}

// ---------------------------------------------------------------- quadtree
struct Nodes2 {
  int *sys, *ij, *begin, *end, *child, *parent;
  uint8_t *depth;
  double *center;
};

__global__ void k2_roots(int nsys, const int64_t *__restrict__ offs, const double *__restrict__ sysbox,
                         Nodes2 na) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  const double *b = sysbox + 6 * s;
  na.sys[s] = s;
  na.ij[2 * s] = na.ij[2 * s + 1] = 0;
  na.depth[s] = 0;
  na.begin[s] = (int)offs[s];
  na.end[s] = (int)offs[s + 1];
  na.child[s] = -1;
  na.parent[s] = -1;
  na.center[2 * s] = node_center_axis(b[0], b[2], 0, 0);
  na.center[2 * s + 1] = node_center_axis(b[1], b[3], 0, 0);
}

// sorted keys (system id above the digits) for subdivide.cuh
struct Keys2 {
  int64_t n;
  const uint64_t *keys;
  int maxbox, maxd;

  // digits that two keys share, -1 in different systems
  static __device__ __forceinline__ int shared(uint64_t a, uint64_t b) {
    const uint64_t v = a ^ b;
    if (v == 0) return kKeyBits;
    if (v >> kSysShift) return -1;
    return (__clzll((long long)v) - (64 - kSysShift)) / 2;
  }
  // depths lo .. hi of the internal nodes that start at place i
  __device__ __forceinline__ void internal_depths(int64_t i, int &lo, int &hi) const {
    lo = kKeyBits + 1;
    hi = -1;
    if (i + maxbox >= n) return;
    const uint64_t k = keys[i];
    lo = i == 0 ? 0 : shared(keys[i - 1], k) + 1;
    hi = min(shared(k, keys[i + maxbox]), maxd - 1);
    if (lo > hi) {
      lo = kKeyBits + 1;
      hi = -1;
    }
  }
};

// every second bit of a key from bit 0
__device__ __forceinline__ int every_second(uint64_t v) {
  v &= 0x5555555555555555ull;
  v = (v | (v >> 1)) & 0x3333333333333333ull;
  v = (v | (v >> 2)) & 0x0f0f0f0f0f0f0f0full;
  v = (v | (v >> 4)) & 0x00ff00ff00ff00ffull;
  v = (v | (v >> 8)) & 0x0000ffff0000ffffull;
  v = (v | (v >> 16)) & 0x00000000ffffffffull;
  return (int)v;
}

// four threads per internal node, thread c making child c: its points end at
// the first key beyond its digits, and begin where child c-1's end
__global__ void k2_make_nodes(int total, LevelStarts ls, const int *__restrict__ start,
                              const int *__restrict__ prank, Keys2 ks, Nodes2 na,
                              const double *__restrict__ sysbox) {
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int c = (int)(g & 3);
  const bool live = (g >> 2) < total;
  const int rk = live ? (int)(g >> 2) : 0;
  int d = 0;
  while (d < kKeyBits - 1 && rk >= ls.rank[d + 1]) ++d;
  const int i = start[rk];
  const uint64_t k = ks.keys[i];
  const int sy = (int)(k >> kSysShift);
  const int shift = 2 * (kKeyBits - d - 1);
  const uint64_t up = k >> (shift + 2), pk = (up << 2) | (uint64_t)c;   // with the system id
  int lo = i;
  int64_t hi = ks.n;
  while (lo < hi) {
    const int mid = (int)((lo + hi) >> 1);
    if ((ks.keys[mid] >> shift) <= pk) lo = mid + 1; else hi = mid;
  }
  // the four threads of a node are four consecutive lanes
  const int prev = __shfl_up_sync(0xffffffffu, lo, 1, 4);
  if (!live) return;
  const int node = d == 0 ? sy : ls.node[d] + 4 * (prank[rk] - ls.rank[d - 1]) + (int)(up & 3);
  const int base = ls.node[d + 1] + 4 * (rk - ls.rank[d]);
  if (c == 0) na.child[node] = base;
  const int cn = base + c, b = c == 0 ? i : prev;
  const double *bx = sysbox + 6 * sy;
  const uint64_t cell = pk & ((1ull << 2 * (d + 1)) - 1);
  const int ci = every_second(cell), cj = every_second(cell >> 1);
  na.sys[cn] = sy;
  na.ij[2 * cn] = ci;
  na.ij[2 * cn + 1] = cj;
  na.depth[cn] = (uint8_t)(d + 1);
  na.begin[cn] = b;
  na.end[cn] = lo;
  if (!(lo - b > ks.maxbox && d + 1 < ks.maxd)) na.child[cn] = -1;   // else its own threads set it
  na.parent[cn] = node;
  na.center[2 * cn] = node_center_axis(bx[0], bx[2], d + 1, ci);
  na.center[2 * cn + 1] = node_center_axis(bx[1], bx[3], d + 1, cj);
}

__global__ void k2_flag(int cnt, int off, const int *__restrict__ begin, const int *__restrict__ end,
                        int maxbox, int d, int maxd, int *__restrict__ flags) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  int c = end[off + i] - begin[off + i];
  flags[i] = (c > maxbox && d < maxd) ? 1 : 0;
}

__global__ void k2_children(int cnt, int off, int child_off, const int *__restrict__ flags,
                            const int *__restrict__ pos, const uint64_t *__restrict__ skeys, int d,
                            Nodes2 na, const double *__restrict__ sysbox) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  int node = off + i;
  if (!flags[i]) {
    na.child[node] = -1;
    return;
  }
  int base = child_off + 4 * pos[i];
  na.child[node] = base;
  int b = na.begin[node], e = na.end[node];
  int shift = 2 * (kKeyBits - d - 1);
  int s = na.sys[node];
  const double *bx = sysbox + 6 * s;
  int pi = na.ij[2 * node], pj = na.ij[2 * node + 1];
  int start = b;
  for (int c = 0; c < 4; ++c) {
    int lo = start, hi = e;
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if ((int)((skeys[mid] >> shift) & 3ull) <= c) lo = mid + 1; else hi = mid;
    }
    int cn = base + c;
    int ci = (pi << 1) | (c & 1), cj = (pj << 1) | ((c >> 1) & 1);
    na.sys[cn] = s;
    na.ij[2 * cn] = ci;
    na.ij[2 * cn + 1] = cj;
    na.depth[cn] = (uint8_t)(d + 1);
    na.begin[cn] = start;
    na.end[cn] = lo;
    na.child[cn] = -1;
    na.parent[cn] = node;
    na.center[2 * cn] = node_center_axis(bx[0], bx[2], d + 1, ci);
    na.center[2 * cn + 1] = node_center_axis(bx[1], bx[3], d + 1, cj);
    start = lo;
  }
}

__device__ __forceinline__ bool adj2(const int *ij, int a, int b) {
  int dx = ij[2 * a] - ij[2 * b], dy = ij[2 * a + 1] - ij[2 * b + 1];
  return dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1;
}

// colleagues of every node in node order, 16 threads per node: thread j < 9 walks
// down from the root of the node's system to the neighbouring cell j, and the
// cells found are placed by counting smaller node numbers (as in tree.cu)
__global__ void k2_colleagues(int nn, const int *__restrict__ begin, const int *__restrict__ end,
                              const int *__restrict__ child, const int *__restrict__ sys,
                              const int *__restrict__ ij, const uint8_t *__restrict__ depth,
                              int *__restrict__ col, int *__restrict__ ncol) {
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int c = (int)(g >> 4), t = (int)(g & 15);
  int q = -1;
  if (c < nn && t < 9 && end[c] > begin[c]) {
    const int d = depth[c];
    const int i = ij[2 * c] + t % 3 - 1, j = ij[2 * c + 1] + t / 3 - 1;
    if (((i | j) & ~((1 << d) - 1)) == 0) {     // inside the box
      q = sys[c];
      for (int b = d - 1; b >= 0 && q >= 0; --b) {
        const int c0 = child[q];
        q = c0 < 0 ? -1 : c0 + (((i >> b) & 1) | ((j >> b) & 1) << 1);
      }
      if (q >= 0 && end[q] == begin[q]) q = -1;
    }
  }
  int at = 0, n = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int o = __shfl_sync(0xffffffffu, q, k, 16);
    if (o >= 0) {
      ++n;
      if (o < q) ++at;
    }
  }
  if (q >= 0) col[9 * c + at] = q;
  if (c < nn && t == 0) ncol[c] = n;
}

// far sources of node t; mode 0 counts, mode 1 writes
__global__ void k2_far(int nn, const int *__restrict__ begin, const int *__restrict__ end,
                       const int *__restrict__ child, const int *__restrict__ parent,
                       const int *__restrict__ ij, const int *__restrict__ col,
                       const int *__restrict__ ncol, int *__restrict__ far_cnt,
                       const int *__restrict__ far_off, int *__restrict__ far_src, int mode) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nn) return;
  int k = 0;
  int w = mode ? far_off[t] : 0;
  int p = parent[t];
  if (end[t] > begin[t] && p >= 0) {
    for (int j = 0; j < ncol[p]; ++j) {
      int c0 = child[col[9 * p + j]];
      if (c0 < 0) continue;
      for (int o = 0; o < 4; ++o) {
        int s = c0 + o;
        if (end[s] == begin[s] || adj2(ij, t, s)) continue;
        if (mode) far_src[w + k] = s;
        ++k;
      }
    }
  }
  if (!mode) far_cnt[t] = k;
}

__global__ void k2_leaf_starts(int nn, const int *__restrict__ begin, const int *__restrict__ end,
                               const int *__restrict__ child, int *__restrict__ flags) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  if (child[i] < 0 && end[i] > begin[i]) flags[begin[i]] = 1;
}

__global__ void k2_leaf_ranges(int nn, int n, const int *__restrict__ begin, const int *__restrict__ end,
                               const int *__restrict__ child, const int *__restrict__ incl,
                               int *__restrict__ lf_begin, int *__restrict__ lf_end,
                               int *__restrict__ leaf_node, int *__restrict__ leaf_be) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  int b = begin[i], e = end[i];
  if (i == 0) leaf_be[incl[n - 1]] = n;          // closes the last leaf
  if (e > b) {
    lf_begin[i] = incl[b] - 1;
    lf_end[i] = incl[e - 1];
    if (child[i] < 0) {
      leaf_node[incl[b] - 1] = i;
      leaf_be[incl[b] - 1] = b;
    }
  } else {
    lf_begin[i] = lf_end[i] = 0;
  }
}

// near leaf-ordinal ranges of leaf L; mode 0 counts (zero for the ordinals from
// the last leaf up to nbound; over: particles of the largest leaf above the
// capacity), mode 1 writes
__global__ void k2_near(int nbound, const int *__restrict__ nleaves_p,
                        const int *__restrict__ leaf_node, const int *__restrict__ begin,
                        const int *__restrict__ end, const int *__restrict__ child,
                        const int *__restrict__ parent, const int *__restrict__ col,
                        const int *__restrict__ ncol, const int *__restrict__ lf_begin,
                        const int *__restrict__ lf_end, int *__restrict__ near_cnt,
                        const int *__restrict__ near_off, int2 *__restrict__ near_rng, int maxbox,
                        int *__restrict__ over, int mode) {
  int L = blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= nbound) return;
  if (L >= *nleaves_p) {
    if (!mode) near_cnt[L] = 0;
    return;
  }
  int node = leaf_node[L];
  if (!mode && end[node] - begin[node] > maxbox) atomicMax(over, end[node] - begin[node]);
  int k = 0;
  int w = mode ? near_off[L] : 0;
  for (int j = 0; j < ncol[node]; ++j) {
    int q = col[9 * node + j];
    if (mode) near_rng[w + k] = make_int2(lf_begin[q], lf_end[q]);
    ++k;
  }
  for (int a = parent[node]; a >= 0; a = parent[a]) {
    for (int j = 0; j < ncol[a]; ++j) {
      int q = col[9 * a + j];
      if (child[q] >= 0 || end[q] == begin[q]) continue;
      if (mode) near_rng[w + k] = make_int2(lf_begin[q], lf_end[q]);
      ++k;
    }
  }
  if (!mode) near_cnt[L] = k;
}

// ------------------------------------------------------------------ passes
// P2M: a_{-i} += q (z - zc)^{i-1}, i = 1..p-1 (arandevelopment2d.c:167-189);
// one warp per leaf, lanes over particles, warp sums per term.
__global__ void k2_p2m(int nleaves, int p, const int *__restrict__ leaf_node,
                       const int *__restrict__ begin, const int *__restrict__ end,
                       const double *__restrict__ center, const double *__restrict__ sx,
                       const double *__restrict__ sy, const double *__restrict__ sq,
                       zd *__restrict__ mult) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= nleaves) return;
  int node = leaf_node[warp];
  int b = begin[node], e = end[node];
  double cx = center[2 * node], cy = center[2 * node + 1];
  zd acc[3];
  for (int k = 0; k < 3; ++k) acc[k] = cmake(0.0, 0.0);
  for (int base = b; base < e; base += 32) {
    int i = base + lane;
    zd d = cmake(0.0, 0.0), tmp = cmake(0.0, 0.0);
    if (i < e) {
      d = cmake(sx[i] - cx, sy[i] - cy);
      tmp = cmake(sq[i], 0.0);
    }
    for (int t = 1; t < p; ++t) {
      double re = shfl_sum(tmp.re), im = shfl_sum(tmp.im);
      if ((t & 31) == lane) {
        zd v = cmake(re, im);
        // constant register indices (no local-memory array)
        if (t < 32) acc[0] = cadd(acc[0], v);
        else if (t < 64) acc[1] = cadd(acc[1], v);
        else acc[2] = cadd(acc[2], v);
      }
      tmp = zmul(tmp, d);
    }
  }
  const int P1 = p + 1;
  for (int k = 0; k < 3; ++k) {
    int t = lane + 32 * k;
    if (t <= p) mult[(int64_t)node * P1 + t] = acc[k];
  }
}

// M2M, one level: warp per node of the level; the children's multipoles
// re-expanded at the node (aran_laurent_seriesd_translate, negative part:
// b_{-i} += sum_{j<i} C(i-1, j-1) a_{-j} (zs - zd)^{i-j} + a_{-i}).
__global__ void k2_m2m(int cnt, int off, int p, const int *__restrict__ child,
                       const int *__restrict__ begin, const int *__restrict__ end,
                       const double *__restrict__ center, const double *__restrict__ binom, int nb,
                       zd *__restrict__ mult) {
  __shared__ zd sm[4][kMaxOrder2d + 1];
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int k = blockIdx.x * (blockDim.x >> 5) + wl;
  int node = off + k;
  bool active = k < cnt && child[node] >= 0;
  const int P1 = p + 1;
  zd acc[3];
  for (int s = 0; s < 3; ++s) acc[s] = cmake(0.0, 0.0);
  if (active) {
    int c0 = child[node];
    double px = center[2 * node], py = center[2 * node + 1];
    for (int c = c0; c < c0 + 4; ++c) {
      if (end[c] == begin[c]) continue;
      __syncwarp();
      for (int t = lane; t <= p; t += 32) sm[wl][t] = mult[(int64_t)c * P1 + t];
      __syncwarp();
      zd z0 = cmake(center[2 * c] - px, center[2 * c + 1] - py);
      for (int s = 0; s < 3; ++s) {
        int i = lane + 32 * s;
        if (i > p) break;
        if (i == 0) {
          acc[s] = cadd(acc[s], sm[wl][0]);
          continue;
        }
        zd sum = cmake(0.0, 0.0);
        for (int j = 1; j < i; ++j) {
          double bc = binom[(i - 1) * nb + (j - 1)];
          sum = zmul(cadd(sum, zscale(sm[wl][j], bc)), z0);
        }
        acc[s] = cadd(acc[s], cadd(sum, sm[wl][i]));
      }
    }
    for (int s = 0; s < 3; ++s) {
      int i = lane + 32 * s;
      if (i <= p) mult[(int64_t)node * P1 + i] = acc[s];
    }
  }
}

// M2L: warp per target node, lanes per local term i:
// L_i += (-1)^i w^i sum_{j=1}^{p-1} C(i+j-1, j-1) a_{-j} w^j, w = 1 / (zt - zs)
// (aran_laurent_seriesd_to_taylor, aranlaurentseriesd.c:409-452).  The FP64
// pipe is the whole cost (half a lane a cycle per scheduler), so the lanes
// take a source each for w, a scan of products makes its powers (five
// complex products) and the terms a_{-j} w^j are shared through shared
// memory: two operations per (i, j) where Horner's rule in every lane took
// six, about 70 a source where it took 175.  60k particles, order 20, leaf
// 32 (137k translations) on GB300: 0.53 ms, 1.52 before.
template <int S>
__global__ void __launch_bounds__(128) k2_m2l(int nn, int p, const int *__restrict__ far_off,
                                              const int *__restrict__ far_src,
                                              const double *__restrict__ center,
                                              const double *__restrict__ binom, int nb,
                                              const zd *__restrict__ mult, zd *__restrict__ loc) {
  extern __shared__ double smem[];
  const int P1 = p + 1;
  const int SP = p | 1;                  // odd row stride: conflict-free lanes
  double *tab = smem;                    // tab[i * SP + j] = C(i+j-1, j-1)
  zd *src = reinterpret_cast<zd *>(smem + ((P1 * SP + 1) & ~1));
  for (int x = threadIdx.x; x < P1 * SP; x += blockDim.x) {
    int i = x / SP, j = x % SP;
    tab[x] = (j >= 1 && j < p) ? binom[(i + j - 1) * nb + (j - 1)] : 0.0;
  }
  __syncthreads();
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int t = blockIdx.x * (blockDim.x >> 5) + wl;
  if (t >= nn) return;
  const int f0 = far_off[t], f1 = far_off[t + 1];
  if (f0 == f1) return;
  zd *ms = src + wl * 32 * S;
  const double tx = center[2 * t], ty = center[2 * t + 1];
  zd acc[S];
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = cmake(0.0, 0.0);
  for (int g = f0; g < f1; g += 32) {
    const int cnt = min(32, f1 - g);
    // lane k: w of source g + k
    int sn = far_src[g + min(lane, cnt - 1)];
    const zd w = zinv(cmake(tx - center[2 * sn], ty - center[2 * sn + 1]));
    for (int k = 0; k < cnt; ++k) {
      const int sk = __shfl_sync(0xffffffffu, sn, k);
      zd a[S];
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int j = lane + 32 * s;
        a[s] = j >= 1 && j < p ? mult[(int64_t)sk * P1 + j] : cmake(0.0, 0.0);
      }
      zd v = cmake(__shfl_sync(0xffffffffu, w.re, k), __shfl_sync(0xffffffffu, w.im, k));
      // lane l: w^(l+1)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const zd u = cmake(__shfl_up_sync(0xffffffffu, v.re, o),
                           __shfl_up_sync(0xffffffffu, v.im, o));
        if (lane >= o) v = zmul(v, u);
      }
      zd wp[S];
      wp[0] = cmake(__shfl_up_sync(0xffffffffu, v.re, 1), __shfl_up_sync(0xffffffffu, v.im, 1));
      if (lane == 0) wp[0] = cmake(1.0, 0.0);
      const zd w32 = cmake(__shfl_sync(0xffffffffu, v.re, 31), __shfl_sync(0xffffffffu, v.im, 31));
#pragma unroll
      for (int s = 1; s < S; ++s) wp[s] = zmul(wp[s - 1], w32);
      __syncwarp();
#pragma unroll
      for (int s = 0; s < S; ++s) ms[lane + 32 * s] = zmul(a[s], wp[s]);
      __syncwarp();
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int i = lane + 32 * s;
        if (i > p) break;
        const double *row = tab + i * SP;
        zd sum = cmake(0.0, 0.0);
        for (int j = p - 1; j >= 1; --j) {      // small terms first, as in Horner's rule
          sum.re = fma(row[j], ms[j].re, sum.re);
          sum.im = fma(row[j], ms[j].im, sum.im);
        }
        acc[s] = cmake(fma(-sum.im, wp[s].im, fma(sum.re, wp[s].re, acc[s].re)),
                       fma(sum.im, wp[s].re, fma(sum.re, wp[s].im, acc[s].im)));
      }
    }
  }
#pragma unroll
  for (int s = 0; s < S; ++s) {
    int i = lane + 32 * s;
    if (i <= p) {
      zd *o = loc + (int64_t)t * P1 + i;
      *o = cadd(*o, (i & 1) ? cmake(-acc[s].re, -acc[s].im) : acc[s]);
    }
  }
}

// L2L, one level: warp per node of the level (depth >= 1); the parent local
// re-expanded at the node (aran_taylor_translate: b_i += sum_{j>=i}
// C(j, i) a_j z^{j-i}, Horner from a_p, z = zchild - zparent).
__global__ void k2_l2l(int cnt, int off, int p, const int *__restrict__ parent,
                       const int *__restrict__ begin, const int *__restrict__ end,
                       const double *__restrict__ center, const double *__restrict__ binom, int nb,
                       zd *__restrict__ loc) {
  __shared__ zd sm[4][kMaxOrder2d + 1];
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int k = blockIdx.x * (blockDim.x >> 5) + wl;
  if (k >= cnt) return;
  int node = off + k;
  int par = parent[node];
  if (par < 0 || end[node] == begin[node]) return;
  const int P1 = p + 1;
  for (int t = lane; t <= p; t += 32) sm[wl][t] = loc[(int64_t)par * P1 + t];
  __syncwarp();
  zd z = cmake(center[2 * node] - center[2 * par], center[2 * node + 1] - center[2 * par + 1]);
  for (int s = 0; s < 3; ++s) {
    int i = lane + 32 * s;
    if (i > p) break;
    zd sum = sm[wl][p];
    for (int j = p - 1; j >= i; --j) sum = cadd(zmul(sum, z), zscale(sm[wl][j], binom[j * nb + i]));
    zd *o = loc + (int64_t)node * P1 + i;
    *o = cadd(*o, sum);
  }
}

// 1 / x in FP64 from the upper word y0 of the hardware approximation (20
// significant bits) by one third-order Newton (Householder) step, y0 + y0 (e
// + e^2) with e = 1 - x y0 rounded once: three FP64 operations, within an ulp
// of the correctly rounded value
__device__ __forceinline__ double rcp_h3(double x) {
  double a;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(a) : "d"(x));
  const double y0 = __hiloint2double(__double2hiint(a), 0);
  const double e = fma(-x, y0, 1.0);
  return fma(y0, fma(e, e, e), y0);
}

// P2P: a block of 128 threads per leaf, every source of the near ranges
// (tests/dummypot.c:62-76, both directions covered by the symmetric lists).
// As in the 3D FP64 near field the FP64 pipe times idle lanes is the cost: a
// leaf of n targets gets floor(128 / n) threads per target, striding over
// the concatenation of its near ranges; 10 FP64 operations a pair (a warp
// per leaf with its targets in the lanes kept 46 % of them busy at 15 points
// a leaf, and the correctly rounded reciprocal took half the operations).
__global__ void __launch_bounds__(128) k2_p2p(int nleaves, const int *__restrict__ leaf_be,
                                              const int *__restrict__ near_off,
                                              const int2 *__restrict__ near_rng,
                                              const double *__restrict__ sx,
                                              const double *__restrict__ sy,
                                              const double *__restrict__ sq,
                                              zd *__restrict__ near_acc) {
  __shared__ zd red[128];
  const int L = blockIdx.x;
  const int b = leaf_be[L], nt = leaf_be[L + 1] - b;
  const int r0 = near_off[L], r1 = near_off[L + 1];
  for (int tb = blockIdx.y * 128; tb < nt; tb += 128 * gridDim.y) {
    const int rem = min(nt - tb, 128);
    const int s = 128 / rem;                  // threads per target
    const int ti = threadIdx.x / s, sub = threadIdx.x - ti * s;
    const bool active = ti < rem;
    const int t = b + tb + (active ? ti : 0);
    double re = 0.0, im = 0.0;
    if (active) {
      const double xi = sx[t], yi = sy[t];
      int rr = r0 - 1, je = 0, j = sub;
      for (;;) {
        bool more = true;
        while (j >= je) {                      // j counts past je: into the next ranges
          if (++rr >= r1) {
            more = false;
            break;
          }
          const int2 rg = near_rng[rr];
          j += leaf_be[rg.x] - je;
          je = leaf_be[rg.y];
        }
        if (!more) break;
        const double dx = xi - sx[j], dy = yi - sy[j];
        const double r2 = dx * dx + dy * dy;
        if (j != t) {
          const unsigned ex = ((unsigned)__double2hiint(r2) >> 20) & 2047u;
          double inv = rcp_h3(r2);
          if (ex - 23u > 2000u) inv = __drcp_rn(r2);
          const double w = sq[j] * inv;
          re = fma(dx, w, re);
          im = fma(-dy, w, im);
        }
        j += s;
      }
    }
    red[threadIdx.x] = cmake(re, im);
    __syncthreads();
    int o = 1;
    while (2 * o < s) o *= 2;
    for (; o > 0 && s > 1; o >>= 1) {
      if (active && sub < o && sub + o < s)
        red[threadIdx.x] = cadd(red[threadIdx.x], red[threadIdx.x + o]);
      __syncthreads();
    }
    if (active && sub == 0) near_acc[t] = red[threadIdx.x];
    __syncthreads();
  }
}

// L2P + near field + unsort: acc[perm[i]] = L(z_i - zc) + near_i
// (aran_laurent_seriesd_evaluate, aranlaurentseriesd.c:311-347, Horner)
__global__ void k2_l2p(int64_t n, int p, const int *__restrict__ incl, const int *__restrict__ leaf_node,
                       const double *__restrict__ center, const double *__restrict__ sx,
                       const double *__restrict__ sy, const zd *__restrict__ loc,
                       const zd *__restrict__ near_acc, const int *__restrict__ perm,
                       double *__restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int node = leaf_node[incl[i] - 1];
  const zd *a = loc + (int64_t)node * (p + 1);
  zd z = cmake(sx[i] - center[2 * node], sy[i] - center[2 * node + 1]);
  zd v = a[p];
  for (int k = p - 1; k >= 0; --k) v = cadd(zmul(v, z), a[k]);
  v = cadd(v, near_acc[i]);
  int o = perm[i];
  out[2 * (int64_t)o] = v.re;
  out[2 * (int64_t)o + 1] = v.im;
}

// ------------------------------------------------- mixed precision passes
// FP32 expansions scaled by the node size h (the larger side of the
// system's box / 2^depth): multipole ma_k = a_{-k} / h^{k-1}, local
// la_k = b_k h^k, so every operator works on O(1) numbers whatever the
// depth; centres and node sizes stay FP64, near-field differences are FP32 hi +
// lo (close ones FP64) with compensated FP32 sums, and every particle's near and far
// parts are added in FP64.  The operators are those of the FP64 kernels
// above with z/h in place of z (rho = h_child / h_parent = 1/2):
//   M2M  mb_i = sum_{j<i} C(i-1, j-1) rho^{j-1} ma_j u^{i-j} + rho^{i-1} ma_i,
//        u = (z_child - z_parent) / h_parent;
//   M2L  la_i = (1/h) (-w)^i sum_j C(i+j-1, j-1) ma_j w^j, w = h / (zt - zs);
//   L2L  lc_i = rho^i sum_{j>=i} C(j, i) lb_j u^{j-i};
//   L2P  sum_k la_k ((z - zc) / h)^k;  P2M  ma_k = sum q ((z - zc) / h)^{k-1}.
typedef cplx<float> zf;

__device__ __forceinline__ double node_size2(const double *__restrict__ sysbox, int sys, int depth) {
  const double *b = sysbox + 6 * sys;
  return fmax(b[2] - b[0], b[3] - b[1]) * ldexp(1.0, -depth);
}

__device__ __forceinline__ float shfl_sumf(float v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ zf zfmul(zf a, zf b) {
  return cmake(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}

__global__ void k2f_p2m(int nleaves, int p, const int *__restrict__ leaf_node,
                        const int *__restrict__ begin, const int *__restrict__ end,
                        const int *__restrict__ sysn, const uint8_t *__restrict__ depth,
                        const double *__restrict__ sysbox, const double *__restrict__ center,
                        const double *__restrict__ sx, const double *__restrict__ sy,
                        const double *__restrict__ sq, zf *__restrict__ mult) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= nleaves) return;
  int node = leaf_node[warp];
  int b = begin[node], e = end[node];
  const double cx = center[2 * node], cy = center[2 * node + 1];
  const double ih = 1.0 / node_size2(sysbox, sysn[node], depth[node]);
  zf acc[3];
  for (int k = 0; k < 3; ++k) acc[k] = cmake(0.f, 0.f);
  for (int base = b; base < e; base += 32) {
    int i = base + lane;
    zf d = cmake(0.f, 0.f), tmp = cmake(0.f, 0.f);
    if (i < e) {
      d = cmake((float)((sx[i] - cx) * ih), (float)((sy[i] - cy) * ih));
      tmp = cmake((float)sq[i], 0.f);
    }
    for (int t = 1; t < p; ++t) {
      float re = shfl_sumf(tmp.re), im = shfl_sumf(tmp.im);
      if ((t & 31) == lane) {
        zf v = cmake(re, im);
        if (t < 32) acc[0] = cadd(acc[0], v);
        else if (t < 64) acc[1] = cadd(acc[1], v);
        else acc[2] = cadd(acc[2], v);
      }
      tmp = zfmul(tmp, d);
    }
  }
  const int P1 = p + 1;
  for (int k = 0; k < 3; ++k) {
    int t = lane + 32 * k;
    if (t <= p) mult[(int64_t)node * P1 + t] = acc[k];
  }
}

__global__ void k2f_m2m(int cnt, int off, int p, const int *__restrict__ child,
                        const int *__restrict__ begin, const int *__restrict__ end,
                        const int *__restrict__ sysn, const uint8_t *__restrict__ depth,
                        const double *__restrict__ sysbox, const double *__restrict__ center,
                        const float *__restrict__ binom, int nb, zf *__restrict__ mult) {
  __shared__ zf sm[4][kMaxOrder2d + 1];
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int k = blockIdx.x * (blockDim.x >> 5) + wl;
  int node = off + k;
  bool active = k < cnt && child[node] >= 0;
  const int P1 = p + 1;
  zf acc[3];
  for (int s = 0; s < 3; ++s) acc[s] = cmake(0.f, 0.f);
  if (active) {
    int c0 = child[node];
    const double px = center[2 * node], py = center[2 * node + 1];
    const double ih = 1.0 / node_size2(sysbox, sysn[node], depth[node]);
    for (int c = c0; c < c0 + 4; ++c) {
      if (end[c] == begin[c]) continue;
      __syncwarp();
      // rho^{t-1} ma_t, rho = 1/2
      for (int t = lane; t <= p; t += 32) {
        const zf v = mult[(int64_t)c * P1 + t];
        const float r = t >= 1 ? ldexpf(1.f, 1 - t) : 1.f;
        sm[wl][t] = cmake(v.re * r, v.im * r);
      }
      __syncwarp();
      const zf u = cmake((float)((center[2 * c] - px) * ih), (float)((center[2 * c + 1] - py) * ih));
      for (int s = 0; s < 3; ++s) {
        int i = lane + 32 * s;
        if (i > p) break;
        if (i == 0) {
          acc[s] = cadd(acc[s], sm[wl][0]);
          continue;
        }
        zf sum = cmake(0.f, 0.f);
        for (int j = 1; j < i; ++j) {
          const float bc = binom[(i - 1) * nb + (j - 1)];
          sum = zfmul(cadd(sum, cmake(sm[wl][j].re * bc, sm[wl][j].im * bc)), u);
        }
        acc[s] = cadd(acc[s], cadd(sum, sm[wl][i]));
      }
    }
    for (int s = 0; s < 3; ++s) {
      int i = lane + 32 * s;
      if (i <= p) mult[(int64_t)node * P1 + i] = acc[s];
    }
  }
}

// M2L, warp per target node, lane i <-> local term i, for orders up to PM.
// Lane k makes w of source k; per source a scan of products makes its powers
// (lane j: w^j) and s_j = ma_j w^j, shared through shared memory
// (double-buffered, so one __syncwarp per source); then
// la_i += (1/h) (-1)^i w^i sum_j C(i+j-1, j-1) s_j with the row of binomials
// in registers and the two parts of s_j in one packed product.  The next
// source's coefficients are loaded while this one runs.  128 systems of order
// 20, 3.4 M translations, on GB300: 0.55 ms; 1.45 with the binomials read from
// shared memory, binary powers in every lane and w made per source.
template <int PM>
__global__ void __launch_bounds__(128) k2f_m2l(int nn, int p, const int *__restrict__ far_off,
                                               const int *__restrict__ far_src,
                                               const int *__restrict__ sysn,
                                               const uint8_t *__restrict__ depth,
                                               const double *__restrict__ sysbox,
                                               const double *__restrict__ center,
                                               const float *__restrict__ binom, int nb,
                                               const zf *__restrict__ mult, zf *__restrict__ loc) {
  constexpr int PE = (PM + 1) & ~1;
  __shared__ __align__(16) uint64_t sbuf[4][2][32];
  const int P1 = p + 1;
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + wl;
  if (t >= nn) return;
  const int f0 = far_off[t], f1 = far_off[t + 1];
  if (f0 == f1) return;
  // row i = lane of the binomials C(i+j-1, j-1), j = 1 .. p-1, each twice
  uint64_t row[PE];
#pragma unroll
  for (int j = 0; j < PE; ++j) {
    const float c = j >= 1 && j < p && lane <= p ? binom[(lane + j - 1) * nb + (j - 1)] : 0.f;
    row[j] = pack2(c, c);
  }
  const double tx = center[2 * t], ty = center[2 * t + 1];
  const double h = node_size2(sysbox, sysn[t], depth[t]), ih = 1.0 / h;
  zf acc = cmake(0.f, 0.f);
  const bool mine = lane >= 1 && lane < p;   // lanes holding a source term
  for (int g = f0; g < f1; g += 32) {
    const int cnt = min(32, f1 - g);
    const int sn = far_src[g + min(lane, cnt - 1)];
    // w = h / (zt - zs): the centre offset in node sizes (small integers,
    // exact in FP32) from FP64, its inverse in FP32
    const float ux = (float)((tx - center[2 * sn]) * ih), uy = (float)((ty - center[2 * sn + 1]) * ih);
    const float iu2 = 1.f / (ux * ux + uy * uy);
    const zf w = cmake(ux * iu2, -uy * iu2);
    int sk = __shfl_sync(0xffffffffu, sn, 0);
    zf ma = mine ? mult[(int64_t)sk * P1 + lane] : cmake(0.f, 0.f);
    for (int k = 0; k < cnt; ++k) {
      zf nma = cmake(0.f, 0.f);
      sk = __shfl_sync(0xffffffffu, sn, k + 1 < cnt ? k + 1 : k);
      if (k + 1 < cnt && mine) nma = mult[(int64_t)sk * P1 + lane];
      // lane l: w^l
      zf v = cmake(__shfl_sync(0xffffffffu, w.re, k), __shfl_sync(0xffffffffu, w.im, k));
      if (lane == 0) v = cmake(1.f, 0.f);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const zf u = cmake(__shfl_up_sync(0xffffffffu, v.re, o),
                           __shfl_up_sync(0xffffffffu, v.im, o));
        if (lane > o) v = zfmul(v, u);
      }
      uint64_t *buf = sbuf[wl][k & 1];
      const zf sj = zfmul(ma, v);
      buf[lane] = pack2(sj.re, sj.im);
      __syncwarp();
      uint64_t sum2 = 0ull, sum3 = 0ull;
#pragma unroll
      for (int j = 0; j < PE; j += 2) {
        const ulonglong2 b2 = *reinterpret_cast<const ulonglong2 *>(buf + j);
        sum2 = fma2(row[j], b2.x, sum2);
        sum3 = fma2(row[j + 1], b2.y, sum3);
      }
      zf sum;
      unpack2(add2(sum2, sum3), sum.re, sum.im);
      acc = cadd(acc, zfmul(sum, v));
      ma = nma;
    }
    __syncwarp();
  }
  // (-1)^i of every term, applied once
  const float ihf = (float)(1.0 / h);
  if (lane <= p) {
    const zf a = (lane & 1) ? cmake(-acc.re, -acc.im) : acc;
    zf *o = loc + (int64_t)t * P1 + lane;
    *o = cadd(*o, cmake(a.re * ihf, a.im * ihf));
  }
}

__global__ void k2f_l2l(int cnt, int off, int p, const int *__restrict__ parent,
                        const int *__restrict__ begin, const int *__restrict__ end,
                        const int *__restrict__ sysn, const uint8_t *__restrict__ depth,
                        const double *__restrict__ sysbox, const double *__restrict__ center,
                        const float *__restrict__ binom, int nb, zf *__restrict__ loc) {
  __shared__ zf sm[4][kMaxOrder2d + 1];
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int k = blockIdx.x * (blockDim.x >> 5) + wl;
  if (k >= cnt) return;
  int node = off + k;
  int par = parent[node];
  if (par < 0 || end[node] == begin[node]) return;
  const int P1 = p + 1;
  for (int t = lane; t <= p; t += 32) sm[wl][t] = loc[(int64_t)par * P1 + t];
  __syncwarp();
  const double ihp = 1.0 / node_size2(sysbox, sysn[par], depth[par]);
  const zf u = cmake((float)((center[2 * node] - center[2 * par]) * ihp),
                     (float)((center[2 * node + 1] - center[2 * par + 1]) * ihp));
  for (int s = 0; s < 3; ++s) {
    int i = lane + 32 * s;
    if (i > p) break;
    zf sum = sm[wl][p];
    for (int j = p - 1; j >= i; --j) {
      const float bc = binom[j * nb + i];
      sum = cadd(zfmul(sum, u), cmake(sm[wl][j].re * bc, sm[wl][j].im * bc));
    }
    const float r = ldexpf(1.f, -i);
    zf *o = loc + (int64_t)node * P1 + i;
    *o = cadd(*o, cmake(sum.re * r, sum.im * r));
  }
}

__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// near field, a block of T threads per target leaf, as the 3D one
// (k_p2p_tile): the concatenated near ranges are staged in tiles of 2 T
// sources as offsets from the leaf's centre (FP32 hi + lo positions), and
// floor(T / n) threads per target sum two sources per packed instruction.
// A pair closer than h/8 (h the target leaf's size), where the offset's
// rounding would show, is left out of the loop and added from the FP64
// positions.  Runs of up to RUN pairs go into Kahan sums, the parts of a target
// are added with compensation: rms error of one-sign sums on leaves of 16, 70 and
// 120 points 1.9e-8, 1.7e-8, 1.5e-8 (one run a tile 2.0e-8, 4.4e-8, 3.9e-8, and the
// kernel 2 to 4 % faster); a warp per leaf, with plain FP32 sums over whole ranges,
// FP64 sums of those and correctly rounded reciprocals, 2.3e-8, 3.6e-8, 4.5e-8.
// Bound by the reciprocal unit (a quarter of a warp per cycle), 8 cycles a pair and
// scheduler, on large leaves, by the blocks' set-up on small ones.
constexpr int k2Ranges = 32;     // near ranges taken together
template <int T>                 // threads, and pairs of a tile
__global__ void __launch_bounds__(T, T == 32 ? 32 : 1280 / T) k2f_p2p(int nleaves, const int *__restrict__ leaf_be,
                        const int *__restrict__ near_off, const int2 *__restrict__ near_rng,
                        const int *__restrict__ leaf_node, const int *__restrict__ sysn,
                        const uint8_t *__restrict__ depth, const double *__restrict__ sysbox,
                        const double *__restrict__ center, const double *__restrict__ sx,
                        const double *__restrict__ sy, const double *__restrict__ sq,
                        const float4 *__restrict__ hl, zd *__restrict__ near_acc) {
  constexpr int RUN = 32;                       // pairs summed plainly
  // pair p of the tile: (-x0, -x1, -y0, -y1) and (q0, q1)
  __shared__ ulonglong2 tA[T];
  __shared__ uint64_t tQ[T];
  __shared__ int tj[2 * T];                     // their particles
  __shared__ int rs[k2Ranges], rp[k2Ranges];    // ranges: first particle, place
  __shared__ int s_tot;
  __shared__ float red[4][T];
  const int L = blockIdx.x;
  const int b = leaf_be[L], nt = leaf_be[L + 1] - b;
  const int r0 = near_off[L], r1 = near_off[L + 1];
  const int node = leaf_node[L];
  const double *box = sysbox + 6 * sysn[node];
  const double cx = center[2 * node] - box[0], cy = center[2 * node + 1] - box[1];
  const float chx = (float)cx, chy = (float)cy;
  const float clx = (float)(cx - (double)chx), cly = (float)(cy - (double)chy);
  const double hh = node_size2(sysbox, sysn[node], depth[node]);
  const float thr2 = (float)(hh * hh / 64.0);
  for (int tb = blockIdx.y * T; tb < nt; tb += T * gridDim.y) {
    const int rem = min(nt - tb, T);
    const int S = T / rem;                      // threads per target
    const int sub = threadIdx.x / rem, ti = threadIdx.x - sub * rem;
    const bool active = sub < S;
    const int t = b + tb + ti;
    const float4 th = hl[t];
    const float tx = (th.x - chx) + (th.z - clx), ty = (th.y - chy) + (th.w - cly);
    const uint64_t tx2 = pack2(tx, tx), ty2 = pack2(ty, ty);
    float ks[2] = {}, kc[2] = {};
    for (int rb = r0; rb < r1; rb += k2Ranges) {
      if (threadIdx.x < k2Ranges) {
        const int rr = rb + threadIdx.x;
        int first = 0, len = 0;
        if (rr < r1) {
          const int2 rg = near_rng[rr];
          first = leaf_be[rg.x];
          len = leaf_be[rg.y] - first;
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (threadIdx.x >= o) incl += v;
        }
        rs[threadIdx.x] = first;
        rp[threadIdx.x] = incl - len;
        if (threadIdx.x == k2Ranges - 1) s_tot = incl;
      }
      __syncthreads();
      const int tot = s_tot;
      for (int k0 = 0; k0 < tot; k0 += 2 * T) {
        const int np = min(T, (tot - k0 + 1) / 2);
        if (threadIdx.x < np) {
          const int k = k0 + 2 * threadIdx.x;
          int g = 0;                            // last range that starts at or before k
#pragma unroll
          for (int o = k2Ranges / 2; o > 0; o >>= 1)
            if (rp[g + o] <= k) g += o;
          float x[2], y[2], q[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (e == 1)
              while (g < k2Ranges - 1 && rp[g + 1] <= k + 1) ++g;
            const bool in = k + e < tot;
            const int j = in ? rs[g] + (k + e - rp[g]) : -1;
            tj[2 * threadIdx.x + e] = j;
            x[e] = 1e18f;                       // no source: no charge, far away
            y[e] = q[e] = 0.f;
            if (in) {
              const float4 v = hl[j];
              x[e] = (chx - v.x) + (clx - v.z);
              y[e] = (chy - v.y) + (cly - v.w);
              q[e] = (float)sq[j];
            }
          }
          tA[threadIdx.x] = make_ulonglong2(pack2(x[0], x[1]), pack2(y[0], y[1]));
          tQ[threadIdx.x] = pack2(q[0], q[1]);
        }
        __syncthreads();
        if (active) {
          unsigned close = 0;   // 1 + pair of the last close pair, above it the one before
          for (int p0 = sub; p0 < np; p0 += RUN * S) {
            const int p1 = min(np, p0 + RUN * S);
            uint64_t p2r = 0ull, p2i = 0ull;
#pragma unroll 2
            for (int p = p0; p < p1; p += S) {
              const ulonglong2 A = tA[p];
              const uint64_t q2 = tQ[p];
              const uint64_t dx = add2(tx2, A.x), dy = add2(ty2, A.y);
              const uint64_t r2 = fma2(dy, dy, mul2(dx, dx));
              float ra, rb2;
              unpack2(r2, ra, rb2);
              const bool ca = ra < thr2, cb = rb2 < thr2;
              if (ca || cb) close = (close << 16) + (unsigned)(p + 1);
              const uint64_t w = mul2(q2, pack2(ca ? 0.f : rcp_ftz(ra), cb ? 0.f : rcp_ftz(rb2)));
              p2r = fma2(dx, w, p2r);
              p2i = fma2(dy, w, p2i);
            }
            float lo, hi;
            unpack2(p2r, lo, hi);
            kahan(ks[0], kc[0], lo + hi);
            unpack2(p2i, lo, hi);
            kahan(ks[1], kc[1], lo + hi);
          }
          if (close) {
            const bool one = close < 65536u;
            for (int p = one ? (int)close - 1 : sub; p < np; p += one ? T : S) {
              const float4 fa = reinterpret_cast<const float4 *>(tA)[p];
              const float2 fq = reinterpret_cast<const float2 *>(tQ)[p];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                float dx = tx + (e ? fa.y : fa.x), dy = ty + (e ? fa.w : fa.z);
                float r2 = fmaf(dy, dy, dx * dx);
                if (!(r2 < thr2)) continue;
                const int j = tj[2 * p + e];
                if (j < 0 || j == t) continue;
                dx = (float)(sx[t] - sx[j]);
                dy = (float)(sy[t] - sy[j]);
                r2 = dx * dx + dy * dy;
                if (!(r2 > 0.f)) continue;
                const float w = (e ? fq.y : fq.x) * __frcp_rn(r2);
                kahan(ks[0], kc[0], dx * w);
                kahan(ks[1], kc[1], dy * w);
              }
            }
          }
        }
        __syncthreads();
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      red[c][threadIdx.x] = ks[c];
      red[2 + c][threadIdx.x] = kc[c];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * rem; i += T) {
      const int tt = i >> 1, c = i & 1;
      float s = red[c][tt], e = -red[2 + c][tt];
      for (int k = 1; k < S; ++k) {
        const float v = red[c][tt + k * rem];
        const float n = s + v, bb = n - s;
        e += ((s - (n - bb)) + (v - bb)) - red[2 + c][tt + k * rem];
        s = n;
      }
      const double v = (double)s + (double)e;
      double *o = reinterpret_cast<double *>(near_acc + b + tb + tt);
      o[c] = c ? -v : v;       // sum of q (dx - i dy) / r^2
    }
    __syncthreads();
  }
}

__global__ void k2f_l2p(int64_t n, int p, const int *__restrict__ incl, const int *__restrict__ leaf_node,
                        const int *__restrict__ sysn, const uint8_t *__restrict__ depth,
                        const double *__restrict__ sysbox, const double *__restrict__ center,
                        const double *__restrict__ sx, const double *__restrict__ sy,
                        const zf *__restrict__ loc, const zd *__restrict__ near_acc,
                        const int *__restrict__ perm, double *__restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int node = leaf_node[incl[i] - 1];
  const zf *a = loc + (int64_t)node * (p + 1);
  const double ih = 1.0 / node_size2(sysbox, sysn[node], depth[node]);
  const zf z = cmake((float)((sx[i] - center[2 * node]) * ih), (float)((sy[i] - center[2 * node + 1]) * ih));
  zf v = a[p];
  for (int k = p - 1; k >= 0; --k) v = cadd(zfmul(v, z), a[k]);
  const zd nr = near_acc[i];
  int o = perm[i];
  out[2 * (int64_t)o] = (double)v.re + nr.re;
  out[2 * (int64_t)o + 1] = (double)v.im + nr.im;
}

// counters: [0] sum cnt_L * sum_r cnt(r), [1] sum cnt_L^2, [2] sum cnt_L (cnt_L + 1) / 2,
// [3] non-empty nodes with a parent
__global__ void k2_stats(int nleaves, int nn, const int *__restrict__ leaf_be,
                         const int *__restrict__ near_off, const int2 *__restrict__ near_rng,
                         const int *__restrict__ begin, const int *__restrict__ end,
                         const int *__restrict__ parent, unsigned long long *__restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long a = 0, b = 0, c = 0, d = 0;
  if (i < nleaves) {
    long long cl = leaf_be[i + 1] - leaf_be[i];
    long long s = 0;
    for (int r = near_off[i]; r < near_off[i + 1]; ++r) {
      int2 rg = near_rng[r];
      s += leaf_be[rg.y] - leaf_be[rg.x];
    }
    a = (unsigned long long)(cl * s);
    b = (unsigned long long)(cl * cl);
    c = (unsigned long long)(cl * (cl + 1) / 2);
  }
  if (i < nn && parent[i] >= 0 && end[i] > begin[i]) d = 1;
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
    d += __shfl_xor_sync(0xffffffffu, d, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, a);
    atomicAdd(out + 1, b);
    atomicAdd(out + 2, c);
    atomicAdd(out + 3, d);
  }
}

}  // namespace
}  // namespace aran

struct AranGpuSolver2d {
  AranGpuConfig2d cfg;
  int device = 0;
  cudaStream_t s0 = nullptr, s1 = nullptr;
  cudaEvent_t ev[2 * aran::Stage::NSTAGE] = {};
  cudaEvent_t ev_lists = nullptr, ev_p2p = nullptr;
  aran::DBuf<double> binom;   // (2p+1)^2 Pascal triangle
  int nb = 0;
  // particles
  aran::DBuf<int64_t> offs;
  aran::DBuf<double> sysbox;
  aran::DBuf<uint64_t> keys_in, keys_out;
  aran::DBuf<int> idx_in, perm, incl, flags;
  aran::DBuf<int> err2;   // input checks of the key pass, largest leaf above the capacity
  int max_leaf = 0;       // no leaf holds more particles
  aran::DBuf<int> internal;   // places and parents of the internal nodes
  int *h_small = nullptr;     // pinned host words for the readbacks
  aran::DBuf<uint8_t> cub_tmp;
  aran::DBuf<double> sx, sy, sq, io_xy, io_q, io_acc;
  aran::DBuf<float4> hl;   // FP32 hi + lo positions in the box (mixed near field)
  // forest
  aran::DBuf<int> nsys_, ij, begin, end, child, parent, col, ncol, far_off, far_src;
  aran::DBuf<int> lf_begin, lf_end, leaf_node, leaf_be, near_off;
  aran::DBuf<int2> near_rng;
  aran::DBuf<uint8_t> depth;
  aran::DBuf<double> center;
  aran::DBuf<aran::cplx<double>> mult, loc, near_acc;
  aran::DBuf<aran::cplx<float>> mult32, loc32;   // mixed precision: scaled FP32 expansions
  aran::DBuf<float> binom32;
  aran::DBuf<unsigned long long> stats_dev;
  std::vector<int> level_off;
  int nnodes = 0, nlevels = 0, nleaves = 0, nrng = 0, empty_roots = 0;
  int64_t n = 0, nfar = 0;
  int64_t stats[11] = {};
  double ms[16] = {};
  int64_t launches = 0;
  // host predicate keeping nodes about to be split as leaves (virtual leaves)
  AranGpuLeafPredicate leaf_pred = nullptr;
  void *leaf_pred_data = nullptr;
  std::vector<double> h_sysbox;   // per system: lbx, lby, ubx, uby, scale x, scale y
};

namespace aran {
namespace {

template <typename T>
void ex_scan(AranGpuSolver2d *s, const T *in, T *out, int n, cudaStream_t st) {
  size_t bytes = 0;
  ACHECK(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, n, st));
  s->cub_tmp.reserve(bytes);
  ACHECK(cub::DeviceScan::ExclusiveSum(s->cub_tmp.ptr, bytes, in, out, n, st));
  s->launches += 2;
}

Nodes2 nodes(AranGpuSolver2d *s) {
  Nodes2 na;
  na.sys = s->nsys_.ptr;
  na.ij = s->ij.ptr;
  na.begin = s->begin.ptr;
  na.end = s->end.ptr;
  na.child = s->child.ptr;
  na.parent = s->parent.ptr;
  na.depth = s->depth.ptr;
  na.center = s->center.ptr;
  return na;
}

void grow(AranGpuSolver2d *s, size_t need, size_t keep, cudaStream_t st) {
  s->nsys_.grow_keep(need, keep, st);
  s->ij.grow_keep(2 * need, 2 * keep, st);
  s->begin.grow_keep(need, keep, st);
  s->end.grow_keep(need, keep, st);
  s->child.grow_keep(need, keep, st);
  s->parent.grow_keep(need, keep, st);
  s->depth.grow_keep(need, keep, st);
  s->center.grow_keep(2 * need, 2 * keep, st);
}

int read_int(const int *d, cudaStream_t st) {
  int h = 0;
  ACHECK(cudaMemcpyAsync(&h, d, sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaStreamSynchronize(st));
  return h;
}

// the nodes of one level about to be split are shown to the host leaf
// predicate (z components 0); those it keeps as leaves lose their flag
void leaf_predicate2(AranGpuSolver2d *s, int off, int cnt, int d, cudaStream_t st) {
  std::vector<int> fl(cnt), b(cnt), e(cnt), ij(2 * (size_t)cnt), sys(cnt);
  ACHECK(cudaMemcpyAsync(fl.data(), s->flags.ptr, cnt * sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(b.data(), s->begin.ptr + off, cnt * sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(e.data(), s->end.ptr + off, cnt * sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(ij.data(), s->ij.ptr + 2 * (size_t)off, 2 * cnt * sizeof(int),
                         cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(sys.data(), s->nsys_.ptr + off, cnt * sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaStreamSynchronize(st));
  bool changed = false;
  for (int i = 0; i < cnt; ++i) {
    if (!fl[i]) continue;
    AranGpuNodeView v;
    std::memset(&v, 0, sizeof(v));
    const double *bx = s->h_sysbox.data() + 6 * (size_t)sys[i];
    for (int a = 0; a < 2; ++a) {
      double lo = bx[a], hi = bx[2 + a];
      for (int bit = d - 1; bit >= 0; --bit) {
        const double mid = (lo + hi) * 0.5;
        if ((ij[2 * (size_t)i + a] >> bit) & 1) lo = mid;
        else hi = mid;
      }
      v.lbound[a] = lo;
      v.ubound[a] = hi;
      v.center[a] = (lo + hi) * 0.5;
    }
    v.point_count = e[i] - b[i];
    v.depth = d;
    if (s->leaf_pred(&v, s->leaf_pred_data)) {
      fl[i] = 0;
      changed = true;
    }
  }
  if (changed)
    ACHECK(cudaMemcpyAsync(s->flags.ptr, fl.data(), cnt * sizeof(int), cudaMemcpyHostToDevice, st));
  ACHECK(cudaStreamSynchronize(st));
}

// the input checks of the key pass
void check_points2(const AranGpuSolver2d *s, int e) {
  if (e & kErrNonFinite) throw InputError{"a particle coordinate or charge is NaN or infinite"};
  if ((e & kErrOutside) && s->cfg.precision == ARAN_PRECISION_MIXED)
    throw InputError{"a particle lies outside its system's box (mixed precision needs every "
                     "point inside it)"};
}

size_t node_estimate2(const AranGpuSolver2d *s, int nsys) {
  return (size_t)nsys + 4 * (s->n / (s->cfg.maxbox + 1) + 1) * 2 + 64;
}

// the quadtrees of the sorted keys, all levels at once (subdivide.cuh): 128
// systems of 1k to 60k particles 0.073 ms, 0.39 level by level; one of 60k 0.057
// ms, 0.36
void subdivide2(AranGpuSolver2d *s, int nsys, cudaStream_t st) {
  const int TB = 256;
  const int64_t n = s->n;
  const int maxd = s->cfg.max_depth > 0 ? s->cfg.max_depth : kKeyBits;
  const int nb = place_blocks(n), nc = kKeyBits * nb;
  s->flags.reserve(2 * (size_t)nc + 2);
  int *first = s->flags.ptr + nc + 1, *hb = s->h_small + 16;
  const Keys2 keys = {n, s->keys_out.ptr, s->cfg.maxbox, maxd};
  count_internal(keys, nb, s->flags.ptr, first, hb,
                 [&](const int *in, int *out, int k) { ex_scan(s, in, out, k, st); }, st);
  s->launches++;
  ACHECK(cudaMemcpyAsync(s->h_small, s->err2.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaStreamSynchronize(st));
  check_points2(s, s->h_small[0]);
  const LevelStarts ls = level_starts(hb, nsys, 4, s->level_off, nullptr);
  s->nlevels = (int)s->level_off.size() - 1;
  s->nnodes = s->level_off.back();
  const int total = hb[kKeyBits];
  grow(s, std::max((size_t)s->nnodes, node_estimate2(s, nsys)), 0, st);
  k2_roots<<<ceil_div(nsys, TB), TB, 0, st>>>(nsys, s->offs.ptr, s->sysbox.ptr, nodes(s));
  ACHECK(cudaGetLastError());
  s->launches++;
  if (total == 0) return;
  s->internal.reserve(2 * (size_t)total);
  int *list = s->internal.ptr;
  k_list_internal<<<nb, kPlaceBlock, 0, st>>>(keys, first, list, list + total);
  ACHECK(cudaGetLastError());
  k2_make_nodes<<<ceil_div(4 * (int64_t)total, TB), TB, 0, st>>>(total, ls, list, list + total, keys,
                                                                 nodes(s), s->sysbox.ptr);
  ACHECK(cudaGetLastError());
  s->launches += 2;
}

// the same level by level, each level's internal nodes shown to the leaf
// predicate before they are split
void subdivide_levels2(AranGpuSolver2d *s, int nsys, cudaStream_t st) {
  const int TB = 256, maxd = s->cfg.max_depth > 0 ? s->cfg.max_depth : kKeyBits;
  check_points2(s, read_int(s->err2.ptr, st));
  grow(s, node_estimate2(s, nsys), 0, st);
  k2_roots<<<ceil_div(nsys, TB), TB, 0, st>>>(nsys, s->offs.ptr, s->sysbox.ptr, nodes(s));
  s->launches++;
  s->level_off.assign(1, 0);
  int off = 0, cnt = nsys, d = 0;
  while (cnt > 0) {
    s->level_off.push_back(off + cnt);
    s->flags.reserve(2 * (size_t)cnt + 2);
    int *pos = s->flags.ptr + cnt + 1;
    k2_flag<<<ceil_div(cnt, TB), TB, 0, st>>>(cnt, off, s->begin.ptr, s->end.ptr, s->cfg.maxbox, d,
                                               maxd, s->flags.ptr);
    s->launches++;
    leaf_predicate2(s, off, cnt, d, st);
    ACHECK(cudaMemsetAsync(s->flags.ptr + cnt, 0, sizeof(int), st));
    ex_scan(s, s->flags.ptr, pos, cnt + 1, st);
    int ninternal = read_int(pos + cnt, st);
    int child_off = off + cnt;
    size_t need = (size_t)child_off + 4 * (size_t)ninternal;
    if (need > s->begin.cap) grow(s, need, child_off, st);
    k2_children<<<ceil_div(cnt, TB), TB, 0, st>>>(cnt, off, child_off, s->flags.ptr, pos,
                                                   s->keys_out.ptr, d, nodes(s), s->sysbox.ptr);
    s->launches++;
    off = child_off;
    cnt = 4 * ninternal;
    ++d;
  }
  s->nnodes = off;
  s->nlevels = d;
}

void build_forest(AranGpuSolver2d *s, int nsys, const double *dxy, const double *dq) {
  cudaStream_t st = s->s0;
  const int TB = 256;
  const int64_t n = s->n;
  s->keys_in.reserve(n);
  s->keys_out.reserve(n);
  s->idx_in.reserve(n);
  s->perm.reserve(n);
  s->err2.reserve(2);
  ACHECK(cudaMemsetAsync(s->err2.ptr, 0, 2 * sizeof(int), st));
  k2_keys<<<ceil_div(n, TB), TB, 0, st>>>(n, nsys, s->offs.ptr, s->sysbox.ptr, dxy, dq,
                                           s->keys_in.ptr, s->idx_in.ptr, s->err2.ptr);
  s->launches++;
  int sysbits = 1;
  while ((1ll << sysbits) < nsys) ++sysbits;
  size_t bytes = 0;
  ACHECK(cub::DeviceRadixSort::SortPairs(nullptr, bytes, s->keys_in.ptr, s->keys_out.ptr,
                                         s->idx_in.ptr, s->perm.ptr, (int)n, 0,
                                         kSysShift + sysbits, st));
  s->cub_tmp.reserve(bytes);
  ACHECK(cub::DeviceRadixSort::SortPairs(s->cub_tmp.ptr, bytes, s->keys_in.ptr, s->keys_out.ptr,
                                         s->idx_in.ptr, s->perm.ptr, (int)n, 0,
                                         kSysShift + sysbits, st));
  s->launches += 4;
  s->sx.reserve(n);
  s->sy.reserve(n);
  s->sq.reserve(n);
  const bool mixed = s->cfg.precision == ARAN_PRECISION_MIXED;
  if (mixed) s->hl.reserve(n);
  k2_gather<<<ceil_div(n, TB), TB, 0, st>>>(n, s->perm.ptr, dxy, dq, s->keys_out.ptr,
                                             s->sysbox.ptr, s->sx.ptr, s->sy.ptr, s->sq.ptr,
                                             mixed ? s->hl.ptr : nullptr);
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::SORT + 1], st));

  if (s->leaf_pred) subdivide_levels2(s, nsys, st);
  else subdivide2(s, nsys, st);
  ACHECK(cudaEventRecord(s->ev[2 * Stage::TREE + 1], st));
}

void build_lists2(AranGpuSolver2d *s) {
  cudaStream_t st = s->s0;
  const int TB = 256;
  const int nn = s->nnodes;
  const int64_t n = s->n;
  s->col.reserve(9 * (size_t)nn);
  s->ncol.reserve(nn);
  k2_colleagues<<<ceil_div(16 * (int64_t)nn, TB), TB, 0, st>>>(nn, s->begin.ptr, s->end.ptr,
                                                               s->child.ptr, s->nsys_.ptr, s->ij.ptr,
                                                               s->depth.ptr, s->col.ptr, s->ncol.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  s->flags.reserve((size_t)std::max<int64_t>(nn, n) + 2);
  s->far_off.reserve(nn + 1);
  k2_far<<<ceil_div(nn, TB), TB, 0, st>>>(nn, s->begin.ptr, s->end.ptr, s->child.ptr, s->parent.ptr,
                                           s->ij.ptr, s->col.ptr, s->ncol.ptr, s->flags.ptr, nullptr,
                                           nullptr, 0);
  s->launches++;
  ACHECK(cudaMemsetAsync(s->flags.ptr + nn, 0, sizeof(int), st));
  ex_scan(s, s->flags.ptr, s->far_off.ptr, nn + 1, st);
  // leaves in key order
  s->incl.reserve(n);
  ACHECK(cudaMemsetAsync(s->flags.ptr, 0, n * sizeof(int), st));
  k2_leaf_starts<<<ceil_div(nn, TB), TB, 0, st>>>(nn, s->begin.ptr, s->end.ptr, s->child.ptr,
                                                   s->flags.ptr);
  s->launches++;
  {
    size_t bytes = 0;
    ACHECK(cub::DeviceScan::InclusiveSum(nullptr, bytes, s->flags.ptr, s->incl.ptr, (int)n, st));
    s->cub_tmp.reserve(bytes);
    ACHECK(cub::DeviceScan::InclusiveSum(s->cub_tmp.ptr, bytes, s->flags.ptr, s->incl.ptr, (int)n, st));
    s->launches += 2;
  }
  // the number of leaves stays on the device until all lists are counted; nlb
  // bounds it
  const int *nleaves_p = s->incl.ptr + n - 1;
  const int nlb = (int)std::min<int64_t>(n, nn);
  s->lf_begin.reserve(nn);
  s->lf_end.reserve(nn);
  s->leaf_node.reserve(nlb + 1);
  s->leaf_be.reserve(nlb + 1);
  k2_leaf_ranges<<<ceil_div(nn, TB), TB, 0, st>>>(nn, (int)n, s->begin.ptr, s->end.ptr, s->child.ptr,
                                                   s->incl.ptr, s->lf_begin.ptr, s->lf_end.ptr,
                                                   s->leaf_node.ptr, s->leaf_be.ptr);
  s->launches++;
  s->near_off.reserve(nlb + 1);
  auto near = [&](int mode) {
    k2_near<<<ceil_div(nlb, TB), TB, 0, st>>>(
        nlb, nleaves_p, s->leaf_node.ptr, s->begin.ptr, s->end.ptr, s->child.ptr, s->parent.ptr,
        s->col.ptr, s->ncol.ptr, s->lf_begin.ptr, s->lf_end.ptr, s->flags.ptr, s->near_off.ptr,
        s->near_rng.ptr, s->cfg.maxbox, s->err2.ptr + 1, mode);
    ACHECK(cudaGetLastError());
    s->launches++;
  };
  near(0);
  ACHECK(cudaMemsetAsync(s->flags.ptr + nlb, 0, sizeof(int), st));
  ex_scan(s, s->flags.ptr, s->near_off.ptr, nlb + 1, st);
  int *hb = s->h_small;
  ACHECK(cudaMemcpyAsync(hb, s->far_off.ptr + nn, sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(hb + 1, nleaves_p, sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(hb + 2, s->near_off.ptr + nlb, sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaMemcpyAsync(hb + 3, s->err2.ptr + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
  ACHECK(cudaStreamSynchronize(st));
  s->nfar = hb[0];
  s->nleaves = hb[1];
  s->nrng = hb[2];
  s->max_leaf = std::max(s->cfg.maxbox, hb[3]);
  s->far_src.reserve(s->nfar + 1);
  k2_far<<<ceil_div(nn, TB), TB, 0, st>>>(nn, s->begin.ptr, s->end.ptr, s->child.ptr, s->parent.ptr,
                                           s->ij.ptr, s->col.ptr, s->ncol.ptr, nullptr, s->far_off.ptr,
                                           s->far_src.ptr, 1);
  s->launches++;
  s->near_rng.reserve(s->nrng + 1);
  near(1);
  ACHECK(cudaEventRecord(s->ev[2 * Stage::LISTS + 1], st));
}

// blocks for a leaf: several for leaves above the capacity, as in 3D (leaf_tiles in
// p2p.cu).  6,000 points within 1e-8, capacity 8: mixed 6 ms, 357 with one block of 32
// threads (327 with a warp per leaf before), FP64 12 ms, 173
int leaf_tiles2(const AranGpuSolver2d *s, int T) {
  return std::min({ceil_div(s->max_leaf, T), 2048 / T, 1 + 100000 / s->nleaves});
}

void run_passes2_mixed(AranGpuSolver2d *s, double *dacc) {
  cudaStream_t st = s->s0, s1 = s->s1;
  const int p = s->cfg.order, P1 = p + 1;
  const int nn = s->nnodes, nl = s->nleaves;
  const int64_t n = s->n;
  typedef cplx<float> zf;
  s->mult32.reserve((size_t)nn * P1);
  s->loc32.reserve((size_t)nn * P1);
  s->near_acc.reserve(n);
  ACHECK(cudaEventRecord(s->ev_lists, st));
  ACHECK(cudaStreamWaitEvent(s1, s->ev_lists, 0));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2P], s1));
  // a warp per leaf up to leaf capacity 64: 64 systems of 1k to 60k particles
  // took 0.25 / 0.26 / 0.39 ms at capacities 20 / 32 / 64 with 32 threads, 0.55
  // / 0.41 / 0.40 with 128; 0.50 and 0.51 at 96.  (The capacity and not the mean
  // occupancy of the batch: a system's bits do not depend on its company.)
  const int T = s->cfg.maxbox <= 64 ? 32 : 128;
  auto p2p = T == 32 ? k2f_p2p<32> : k2f_p2p<128>;
  p2p<<<dim3(nl, leaf_tiles2(s, T)), T, 0, s1>>>(nl, s->leaf_be.ptr, s->near_off.ptr, s->near_rng.ptr,
                                 s->leaf_node.ptr, s->nsys_.ptr, s->depth.ptr, s->sysbox.ptr,
                                 s->center.ptr, s->sx.ptr, s->sy.ptr, s->sq.ptr, s->hl.ptr,
                                 s->near_acc.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2P + 1], s1));
  ACHECK(cudaEventRecord(s->ev_p2p, s1));

  ACHECK(cudaMemsetAsync(s->mult32.ptr, 0, (size_t)nn * P1 * sizeof(zf), st));
  ACHECK(cudaMemsetAsync(s->loc32.ptr, 0, (size_t)nn * P1 * sizeof(zf), st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2M], st));
  k2f_p2m<<<ceil_div((int64_t)nl * 32, 128), 128, 0, st>>>(
      nl, p, s->leaf_node.ptr, s->begin.ptr, s->end.ptr, s->nsys_.ptr, s->depth.ptr, s->sysbox.ptr,
      s->center.ptr, s->sx.ptr, s->sy.ptr, s->sq.ptr, s->mult32.ptr);
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2M + 1], st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2M], st));
  for (int d = s->nlevels - 2; d >= 0; --d) {
    int off = s->level_off[d], cnt = s->level_off[d + 1] - off;
    k2f_m2m<<<ceil_div(cnt, 4), 128, 0, st>>>(cnt, off, p, s->child.ptr, s->begin.ptr, s->end.ptr,
                                              s->nsys_.ptr, s->depth.ptr, s->sysbox.ptr,
                                              s->center.ptr, s->binom32.ptr, s->nb, s->mult32.ptr);
    s->launches++;
  }
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2M + 1], st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2L], st));
  {
    // the instance whose row of binomials is the shortest that holds the order
    auto kern = p <= 12 ? k2f_m2l<12> : (p <= 20 ? k2f_m2l<20> : k2f_m2l<31>);
    kern<<<ceil_div(nn, 4), 128, 0, st>>>(nn, p, s->far_off.ptr, s->far_src.ptr, s->nsys_.ptr,
                                          s->depth.ptr, s->sysbox.ptr, s->center.ptr,
                                          s->binom32.ptr, s->nb, s->mult32.ptr, s->loc32.ptr);
    ACHECK(cudaGetLastError());
    s->launches++;
  }
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2L + 1], st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2L], st));
  for (int d = 2; d < s->nlevels; ++d) {
    int off = s->level_off[d], cnt = s->level_off[d + 1] - off;
    k2f_l2l<<<ceil_div(cnt, 4), 128, 0, st>>>(cnt, off, p, s->parent.ptr, s->begin.ptr, s->end.ptr,
                                              s->nsys_.ptr, s->depth.ptr, s->sysbox.ptr,
                                              s->center.ptr, s->binom32.ptr, s->nb, s->loc32.ptr);
    s->launches++;
  }
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2L + 1], st));
  ACHECK(cudaStreamWaitEvent(st, s->ev_p2p, 0));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2P], st));
  k2f_l2p<<<ceil_div(n, 256), 256, 0, st>>>(n, p, s->incl.ptr, s->leaf_node.ptr, s->nsys_.ptr,
                                            s->depth.ptr, s->sysbox.ptr, s->center.ptr, s->sx.ptr,
                                            s->sy.ptr, s->loc32.ptr, s->near_acc.ptr, s->perm.ptr,
                                            dacc);
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2P + 1], st));
}

void run_passes2(AranGpuSolver2d *s, double *dacc) {
  cudaStream_t st = s->s0, s1 = s->s1;
  const int p = s->cfg.order, P1 = p + 1;
  const int nn = s->nnodes, nl = s->nleaves;
  const int64_t n = s->n;
  if (s->cfg.precision == ARAN_PRECISION_MIXED) {
    run_passes2_mixed(s, dacc);
  } else {
  s->mult.reserve((size_t)nn * P1);
  s->loc.reserve((size_t)nn * P1);
  s->near_acc.reserve(n);
  // near field on its own stream
  ACHECK(cudaEventRecord(s->ev_lists, st));
  ACHECK(cudaStreamWaitEvent(s1, s->ev_lists, 0));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2P], s1));
  k2_p2p<<<dim3(nl, leaf_tiles2(s, 128)), 128, 0, s1>>>(nl, s->leaf_be.ptr, s->near_off.ptr, s->near_rng.ptr, s->sx.ptr,
                             s->sy.ptr, s->sq.ptr, s->near_acc.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2P + 1], s1));
  ACHECK(cudaEventRecord(s->ev_p2p, s1));

  ACHECK(cudaMemsetAsync(s->mult.ptr, 0, (size_t)nn * P1 * sizeof(zd), st));
  ACHECK(cudaMemsetAsync(s->loc.ptr, 0, (size_t)nn * P1 * sizeof(zd), st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2M], st));
  k2_p2m<<<ceil_div((int64_t)nl * 32, 128), 128, 0, st>>>(nl, p, s->leaf_node.ptr, s->begin.ptr,
                                                          s->end.ptr, s->center.ptr, s->sx.ptr,
                                                          s->sy.ptr, s->sq.ptr, s->mult.ptr);
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::P2M + 1], st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2M], st));
  for (int d = s->nlevels - 2; d >= 0; --d) {
    int off = s->level_off[d], cnt = s->level_off[d + 1] - off;
    k2_m2m<<<ceil_div(cnt, 4), 128, 0, st>>>(cnt, off, p, s->child.ptr, s->begin.ptr, s->end.ptr,
                                             s->center.ptr, s->binom.ptr, s->nb, s->mult.ptr);
    s->launches++;
  }
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2M + 1], st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2L], st));
  {
    const int S = (P1 + 31) / 32;        // terms per lane
    const size_t smem = (size_t)((P1 * (p | 1) + 1) & ~1) * sizeof(double) + 4 * 32 * S * sizeof(zd);
    auto kern = S == 1 ? k2_m2l<1> : (S == 2 ? k2_m2l<2> : k2_m2l<3>);
    smem_opt_in(kern, smem);
    kern<<<ceil_div(nn, 4), 128, smem, st>>>(nn, p, s->far_off.ptr, s->far_src.ptr, s->center.ptr,
                                             s->binom.ptr, s->nb, s->mult.ptr, s->loc.ptr);
    ACHECK(cudaGetLastError());
    s->launches++;
  }
  ACHECK(cudaEventRecord(s->ev[2 * Stage::M2L + 1], st));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2L], st));
  for (int d = 2; d < s->nlevels; ++d) {
    int off = s->level_off[d], cnt = s->level_off[d + 1] - off;
    k2_l2l<<<ceil_div(cnt, 4), 128, 0, st>>>(cnt, off, p, s->parent.ptr, s->begin.ptr, s->end.ptr,
                                             s->center.ptr, s->binom.ptr, s->nb, s->loc.ptr);
    s->launches++;
  }
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2L + 1], st));
  ACHECK(cudaStreamWaitEvent(st, s->ev_p2p, 0));
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2P], st));
  k2_l2p<<<ceil_div(n, 256), 256, 0, st>>>(n, p, s->incl.ptr, s->leaf_node.ptr, s->center.ptr,
                                           s->sx.ptr, s->sy.ptr, s->loc.ptr, s->near_acc.ptr,
                                           s->perm.ptr, dacc);
  s->launches++;
  ACHECK(cudaEventRecord(s->ev[2 * Stage::L2P + 1], st));
  }
  // counters
  s->stats_dev.reserve(4);
  ACHECK(cudaMemsetAsync(s->stats_dev.ptr, 0, 4 * sizeof(unsigned long long), st));
  int m = std::max(nl, nn);
  k2_stats<<<ceil_div(m, 256), 256, 0, st>>>(nl, nn, s->leaf_be.ptr, s->near_off.ptr, s->near_rng.ptr,
                                             s->begin.ptr, s->end.ptr, s->parent.ptr, s->stats_dev.ptr);
  s->launches++;
}

int check2(const AranGpuConfig2d *c) {
  if (!c) return fail(ARAN_ERR_INVALID, "config is NULL");
  if (c->maxbox < 1) return fail(ARAN_ERR_INVALID, "maxbox must be >= 1");
  if (c->order < 1 || c->order > kMaxOrder2d)
    return fail(ARAN_ERR_INVALID, "order must be in [1, " + std::to_string(kMaxOrder2d) + "]");
  if (c->max_depth < 0 || c->max_depth > kKeyBits)
    return fail(ARAN_ERR_INVALID, "max_depth must be in [0, 21]");
  if (c->precision != ARAN_PRECISION_FP64 && c->precision != ARAN_PRECISION_MIXED)
    return fail(ARAN_ERR_INVALID, "unknown precision");
  if (c->precision == ARAN_PRECISION_MIXED && c->order > 31)
    return fail(ARAN_ERR_INVALID, "mixed precision 2D solves take orders up to 31");
  return ARAN_OK;
}

}  // namespace
}  // namespace aran

using namespace aran;

extern "C" {

int aran_gpu_solver2d_create(const AranGpuConfig2d *cfg, AranGpuSolver2d **out) {
  if (!out) return fail(ARAN_ERR_INVALID, "out is NULL");
  *out = nullptr;
  int rc = check2(cfg);
  if (rc != ARAN_OK) return rc;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0)
    return fail(ARAN_ERR_NO_DEVICE, std::string("no CUDA device available: ") + cudaGetErrorString(e));
  AranGpuSolver2d *s = new AranGpuSolver2d();
  s->cfg = *cfg;
  try {
    ACHECK(cudaGetDevice(&s->device));
    ACHECK(cudaStreamCreateWithFlags(&s->s0, cudaStreamNonBlocking));
    ACHECK(cudaStreamCreateWithFlags(&s->s1, cudaStreamNonBlocking));
    ACHECK(cudaHostAlloc(&s->h_small, 64 * sizeof(int), cudaHostAllocDefault));
    for (auto &ev : s->ev) ACHECK(cudaEventCreate(&ev));
    ACHECK(cudaEventCreateWithFlags(&s->ev_lists, cudaEventDisableTiming));
    ACHECK(cudaEventCreateWithFlags(&s->ev_p2p, cudaEventDisableTiming));
    // Pascal triangle in doubles (aran/aranbinomial.c:44-51)
    const int p = cfg->order;
    s->nb = 2 * p + 2;
    std::vector<double> b((size_t)s->nb * s->nb, 0.0);
    for (int i = 0; i < s->nb; ++i)
      for (int j = 0; j <= i; ++j)
        b[(size_t)i * s->nb + j] =
            (j == 0 || j == i) ? 1.0 : b[(size_t)(i - 1) * s->nb + j] + b[(size_t)(i - 1) * s->nb + j - 1];
    s->binom.reserve(b.size());
    ACHECK(cudaMemcpyAsync(s->binom.ptr, b.data(), b.size() * sizeof(double), cudaMemcpyHostToDevice,
                           s->s0));
    std::vector<float> bf(b.begin(), b.end());
    s->binom32.reserve(bf.size());
    ACHECK(cudaMemcpyAsync(s->binom32.ptr, bf.data(), bf.size() * sizeof(float),
                           cudaMemcpyHostToDevice, s->s0));
    ACHECK(cudaStreamSynchronize(s->s0));
  } catch (const CudaError &ce) {
    int r = from_cuda(ce);
    aran_gpu_solver2d_destroy(s);
    return r;
  }
  *out = s;
  return ARAN_OK;
}

void aran_gpu_solver2d_destroy(AranGpuSolver2d *s) {
  if (!s) return;
  cudaSetDevice(s->device);
  if (s->s0) cudaStreamSynchronize(s->s0);
  if (s->s1) cudaStreamSynchronize(s->s1);
  s->binom.release();
  s->offs.release();
  s->sysbox.release();
  s->keys_in.release();
  s->keys_out.release();
  s->idx_in.release();
  s->err2.release();
  s->internal.release();
  if (s->h_small) cudaFreeHost(s->h_small);
  s->perm.release();
  s->incl.release();
  s->flags.release();
  s->cub_tmp.release();
  s->sx.release();
  s->sy.release();
  s->sq.release();
  s->hl.release();
  s->io_xy.release();
  s->io_q.release();
  s->io_acc.release();
  s->nsys_.release();
  s->ij.release();
  s->begin.release();
  s->end.release();
  s->child.release();
  s->parent.release();
  s->col.release();
  s->ncol.release();
  s->far_off.release();
  s->far_src.release();
  s->lf_begin.release();
  s->lf_end.release();
  s->leaf_node.release();
  s->leaf_be.release();
  s->near_off.release();
  s->near_rng.release();
  s->depth.release();
  s->center.release();
  s->mult.release();
  s->loc.release();
  s->near_acc.release();
  s->mult32.release();
  s->loc32.release();
  s->binom32.release();
  s->stats_dev.release();
  for (auto &ev : s->ev)
    if (ev) cudaEventDestroy(ev);
  if (s->ev_lists) cudaEventDestroy(s->ev_lists);
  if (s->ev_p2p) cudaEventDestroy(s->ev_p2p);
  if (s->s0) cudaStreamDestroy(s->s0);
  if (s->s1) cudaStreamDestroy(s->s1);
  delete s;
}

int aran_gpu_solver2d_solve(AranGpuSolver2d *s, int nsys, const int64_t *offs, const double *box,
                            const double *xy, const double *q, double *acc, int mem) {
  if (!acc) return fail(ARAN_ERR_INVALID, "NULL argument");
  return aran::solve2d_impl(s, nsys, offs, box, xy, q, acc, mem, false);
}

int aran_gpu_solver2d_set_leaf_predicate(AranGpuSolver2d *s, AranGpuLeafPredicate pred,
                                         void *user_data) {
  if (!s) return fail(ARAN_ERR_INVALID, "solver is NULL");
  s->leaf_pred = pred;
  s->leaf_pred_data = pred ? user_data : nullptr;
  return ARAN_OK;
}

}  // extern "C"

namespace aran {

int solve2d_impl(AranGpuSolver2d *s, int nsys, const int64_t *offs, const double *box,
                 const double *xy, const double *q, double *acc, int mem, bool tree_only) {
  if (!s) return fail(ARAN_ERR_INVALID, "solver is NULL");
  if (nsys < 1 || nsys > (1 << 21)) return fail(ARAN_ERR_INVALID, "nsys must be in [1, 2^21]");
  if (!offs || !box || !xy || !q) return fail(ARAN_ERR_INVALID, "NULL argument");
  if (mem != ARAN_MEM_HOST && mem != ARAN_MEM_DEVICE) return fail(ARAN_ERR_INVALID, "bad mem kind");
  if (offs[0] != 0) return fail(ARAN_ERR_INVALID, "offs[0] must be 0");
  int empty = 0;
  std::vector<double> sb(6 * (size_t)nsys);
  for (int i = 0; i < nsys; ++i) {
    if (offs[i + 1] < offs[i]) return fail(ARAN_ERR_INVALID, "offs must be non-decreasing");
    empty += offs[i + 1] == offs[i];
    for (int a = 0; a < 2; ++a) {
      double lo = box[4 * i + a], hi = box[4 * i + 2 + a];
      if (!(hi > lo) || !std::isfinite(lo) || !std::isfinite(hi))
        return fail(ARAN_ERR_INVALID, "box of system " + std::to_string(i) + " must satisfy lb < ub");
      sb[6 * i + a] = lo;
      sb[6 * i + 2 + a] = hi;
      sb[6 * i + 4 + a] = (double)(1 << kKeyBits) / (hi - lo);
    }
  }
  const int64_t n = offs[nsys];
  if (n < 1) return fail(ARAN_ERR_INVALID, "no particles");
  if (n > (int64_t)1 << 30) return fail(ARAN_ERR_INVALID, "more than 2^30 particles");
  try {
    ACHECK(cudaSetDevice(s->device));
    s->launches = 0;
    s->n = n;
    s->empty_roots = empty;
    cudaStream_t st = s->s0;
    ACHECK(cudaEventRecord(s->ev[2 * Stage::TOTAL], st));
    ACHECK(cudaEventRecord(s->ev[2 * Stage::H2D], st));
    s->offs.reserve(nsys + 1);
    s->sysbox.reserve(sb.size());
    ACHECK(cudaMemcpyAsync(s->offs.ptr, offs, (nsys + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    ACHECK(cudaMemcpyAsync(s->sysbox.ptr, sb.data(), sb.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    const double *dxy = xy, *dq = q;
    double *dacc = acc;
    if (mem == ARAN_MEM_HOST) {
      s->io_xy.reserve(2 * n);
      s->io_q.reserve(n);
      s->io_acc.reserve(2 * n);
      ACHECK(cudaMemcpyAsync(s->io_xy.ptr, xy, 2 * n * sizeof(double), cudaMemcpyHostToDevice, st));
      ACHECK(cudaMemcpyAsync(s->io_q.ptr, q, n * sizeof(double), cudaMemcpyHostToDevice, st));
      dxy = s->io_xy.ptr;
      dq = s->io_q.ptr;
      dacc = s->io_acc.ptr;
    }
    ACHECK(cudaEventRecord(s->ev[2 * Stage::H2D + 1], st));
    ACHECK(cudaEventRecord(s->ev[2 * Stage::SORT], st));
    s->h_sysbox = sb;
    build_forest(s, nsys, dxy, dq);
    if (tree_only) {
      ACHECK(cudaStreamSynchronize(st));
      return ARAN_OK;
    }
    build_lists2(s);
    run_passes2(s, dacc);
    ACHECK(cudaEventRecord(s->ev[2 * Stage::D2H], st));
    if (mem == ARAN_MEM_HOST)
      ACHECK(cudaMemcpyAsync(acc, dacc, 2 * n * sizeof(double), cudaMemcpyDeviceToHost, st));
    unsigned long long cnt[4];
    ACHECK(cudaMemcpyAsync(cnt, s->stats_dev.ptr, sizeof(cnt), cudaMemcpyDeviceToHost, st));
    ACHECK(cudaEventRecord(s->ev[2 * Stage::D2H + 1], st));
    ACHECK(cudaEventRecord(s->ev[2 * Stage::TOTAL + 1], st));
    ACHECK(cudaStreamSynchronize(st));
    ACHECK(cudaStreamSynchronize(s->s1));
    ACHECK(cudaGetLastError());
    std::memset(s->stats, 0, sizeof(s->stats));
    s->stats[0] = s->nnodes - s->empty_roots;
    s->stats[1] = (int64_t)((cnt[0] - cnt[1]) / 2 + cnt[2]);
    s->stats[2] = n;
    s->stats[3] = (int64_t)cnt[3];
    s->stats[4] = s->nfar;
    s->stats[5] = (int64_t)cnt[3];
    s->stats[6] = n;
    auto el = [&](int a, int b) {
      float m = 0.f;
      cudaEventElapsedTime(&m, s->ev[a], s->ev[b]);
      return (double)m;
    };
    s->ms[0] = el(2 * Stage::TOTAL, 2 * Stage::TOTAL + 1);
    s->ms[1] = el(2 * Stage::SORT, 2 * Stage::SORT + 1);
    s->ms[2] = el(2 * Stage::SORT + 1, 2 * Stage::TREE + 1);
    s->ms[3] = el(2 * Stage::TREE + 1, 2 * Stage::LISTS + 1);
    s->ms[4] = el(2 * Stage::P2M, 2 * Stage::P2M + 1);
    s->ms[5] = el(2 * Stage::M2M, 2 * Stage::M2M + 1);
    s->ms[6] = el(2 * Stage::M2L, 2 * Stage::M2L + 1);
    s->ms[7] = el(2 * Stage::L2L, 2 * Stage::L2L + 1);
    s->ms[8] = el(2 * Stage::L2P, 2 * Stage::L2P + 1);
    s->ms[9] = el(2 * Stage::P2P, 2 * Stage::P2P + 1);
    s->ms[10] = el(2 * Stage::H2D, 2 * Stage::H2D + 1);
    s->ms[11] = el(2 * Stage::D2H, 2 * Stage::D2H + 1);
  } catch (const CudaError &ce) {
    return from_cuda(ce);
  } catch (const InputError &ie) {
    // stopped after the key pass: nothing was written
    cudaStreamSynchronize(s->s0);
    cudaStreamSynchronize(s->s1);
    return fail(ARAN_ERR_INVALID, ie.msg);
  }
  return ARAN_OK;
}

int forest2d_to_host(AranGpuSolver2d *s, Forest2dHost &h, bool expansions) {
  try {
    ACHECK(cudaSetDevice(s->device));
    const int nn = s->nnodes;
    h.p = s->cfg.order;
    h.nnodes = nn;
    h.begin.resize(nn);
    h.end.resize(nn);
    h.child.resize(nn);
    h.parent.resize(nn);
    h.sys.resize(nn);
    h.ij.resize(2 * (size_t)nn);
    h.depth.resize(nn);
    h.center.resize(2 * (size_t)nn);
    h.perm.resize(s->n);
    h.sysbox = s->h_sysbox;
    ACHECK(cudaMemcpy(h.begin.data(), s->begin.ptr, nn * sizeof(int), cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.end.data(), s->end.ptr, nn * sizeof(int), cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.child.data(), s->child.ptr, nn * sizeof(int), cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.parent.data(), s->parent.ptr, nn * sizeof(int), cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.sys.data(), s->nsys_.ptr, nn * sizeof(int), cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.ij.data(), s->ij.ptr, 2 * (size_t)nn * sizeof(int), cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.depth.data(), s->depth.ptr, nn, cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.center.data(), s->center.ptr, 2 * (size_t)nn * sizeof(double),
                      cudaMemcpyDeviceToHost));
    ACHECK(cudaMemcpy(h.perm.data(), s->perm.ptr, s->n * sizeof(int), cudaMemcpyDeviceToHost));
    h.mult.clear();
    h.loc.clear();
    if (expansions) {
      const size_t len = (size_t)nn * (h.p + 1) * 2;
      h.mult.resize(len);
      h.loc.resize(len);
      if (s->cfg.precision == ARAN_PRECISION_MIXED) {
        // back from the scaled FP32 storage: a_{-k} = ma_k h^{k-1}, b_k = la_k h^-k
        std::vector<float> m32(len), l32(len);
        ACHECK(cudaMemcpy(m32.data(), s->mult32.ptr, len * sizeof(float), cudaMemcpyDeviceToHost));
        ACHECK(cudaMemcpy(l32.data(), s->loc32.ptr, len * sizeof(float), cudaMemcpyDeviceToHost));
        for (int i = 0; i < nn; ++i) {
          const double *b = s->h_sysbox.data() + 6 * (size_t)h.sys[i];
          const double hs = std::max(b[2] - b[0], b[3] - b[1]) * std::ldexp(1.0, -(int)h.depth[i]);
          for (int k = 0; k <= h.p; ++k) {
            const size_t o = 2 * ((size_t)i * (h.p + 1) + k);
            const double fm = k >= 1 ? std::pow(hs, k - 1) : 1.0, fl = std::pow(hs, -k);
            h.mult[o] = m32[o] * fm;
            h.mult[o + 1] = m32[o + 1] * fm;
            h.loc[o] = l32[o] * fl;
            h.loc[o + 1] = l32[o + 1] * fl;
          }
        }
      } else {
        ACHECK(cudaMemcpy(h.mult.data(), s->mult.ptr, len * sizeof(double), cudaMemcpyDeviceToHost));
        ACHECK(cudaMemcpy(h.loc.data(), s->loc.ptr, len * sizeof(double), cudaMemcpyDeviceToHost));
      }
    }
  } catch (const CudaError &ce) {
    return from_cuda(ce);
  }
  return ARAN_OK;
}

}  // namespace aran

extern "C" {

int aran_gpu_solver2d_get_stats(AranGpuSolver2d *s, int64_t stats[11]) {
  if (!s || !stats) return fail(ARAN_ERR_INVALID, "NULL argument");
  std::memcpy(stats, s->stats, sizeof(s->stats));
  return ARAN_OK;
}

int aran_gpu_solver2d_timings(AranGpuSolver2d *s, double ms[16]) {
  if (!s || !ms) return fail(ARAN_ERR_INVALID, "NULL argument");
  std::memcpy(ms, s->ms, sizeof(s->ms));
  return ARAN_OK;
}

int aran_gpu_solver2d_tree_info(AranGpuSolver2d *s, int64_t info[5]) {
  if (!s || !info) return fail(ARAN_ERR_INVALID, "NULL argument");
  info[0] = s->nnodes;
  info[1] = s->nfar;
  info[2] = s->nrng;
  info[3] = s->nleaves;
  info[4] = s->nlevels > 0 ? s->nlevels - 1 : 0;
  return ARAN_OK;
}

int64_t aran_gpu_solver2d_launches(AranGpuSolver2d *s) { return s ? s->launches : -1; }

}  // extern "C"
