// m2l_fp64.cu -- the FP64 M2L (far_func, aran/aransolver3d.c:333-354, with the
// "point and shoot" operator of aran_spherical_seriesd_to_local_rotate,
// aran/aransphericalseriesd-rotate.c:165-207).
//
// The FP64 pipe takes half a lane per cycle and scheduler: its instructions
// times the lanes they leave idle are the whole cost, loads and index
// arithmetic come free.  So
//  * every stage (rotation to the axis, translation along it, rotation back) is
//    a list of dot products, one per real number it makes: a coefficient's real
//    part, and its imaginary part where that is not zero by itself (the odd
//    blocks have no row or column 0).  The products are sorted by length and
//    dealt to the lanes 32 at a time, so the lanes of a round run equally long
//    (87 to 92 % of them busy at order 12; lanes over coefficients, each making
//    both parts as in the sibling kernel of m2l.cu, kept 65 to 78 %);
//  * an offset d and its opposite share the rotation: with y and y' the rotated
//    sources, z(j) = sum_n V(j, n) (y(n) + (-1)^{j+n} y'(n)), so the even degrees
//    come from u = y + (-1)^n y', the odd ones from w = y - (-1)^n y', and one
//    translation and one rotation back serve two sources.  A child's sources
//    lie at 189 offsets, 49 opposite pairs and 91 alone;
//  * child w walks child 0's offsets through the mirror images (m2l_lanes.cuh), so
//    140 tables serve all children and the warps of a CTA (the eight children
//    of a parent) read the same table at about the same time.  Tables are
//    streamed from L2 in the order the lanes use them: [round][step][lane].
//
// A target's sum is the sum of fixed segments of the units (offsets or pairs), each
// summed on its own and added in order, so a system's bits do not depend on what else
// is solved.  In passes of few parents a CTA takes one segment of a parent and
// leaves its sum in a workspace, in passes of many it takes them all.
// Measured on GB300 against the sibling kernel in FP64: 200k Plummer particles
// at order 12, the whole solve with the near field beside it on the same pipe,
// 40.2 ms, 48.4 before (42.0 with two CTAs an SM); eight served requests, two of
// them in FP64 at order 26, 13.9 ms, 35 before (with the P2M and L2P of
// leaf_fp64.cu).  60k Plummer particles, this kernel alone: 3.8 ms, the FP64 pipe
// active 92 % of the cycles.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "internal.cuh"

namespace aran {

namespace {

constexpr int kF64Warps = 8;
constexpr int kF64Segs = 16;               // segments of the units

// first unit of a segment
__device__ __forceinline__ int seg_unit(int seg, int nunits) {
  return (seg * nunits + kF64Segs - 1) / kF64Segs;
}

// one dot product of a stage: first source and destination in the planes of
// the stage's vectors, length, first step between sources (it grows by one per
// term in the translation, is one in the rotations)
struct F64Task {
  uint16_t src, dst;
  uint8_t cnt, step, flag, pad;   // flag: bit 0 odd degree j, bit 1 imaginary part
};

// task lists and round lengths of order p
struct HostSched {
  M2lFp64Sched d;
  std::vector<F64Task> task;      // [round][lane]
  std::vector<int> trip, toff;    // per round: steps, first entry within the unit's table
  std::vector<int4> gen;          // per task: stage, (l or j), (m' or m), part
};

HostSched make_sched(int p) {
  HostSched h;
  const int nm = tri(p), nl = tri(p + 1);
  int off = 0;
  for (int st = 0; st < 3; ++st) {
    struct T { F64Task t; int4 g; };
    std::vector<T> v;
    const int L = st == 0 ? p : p + 1;
    const int ns = st == 2 ? nl : nm, nd = st == 0 ? nm : nl;   // plane lengths in, out
    for (int l = 0; l < L; ++l)
      for (int m = 0; m <= l; ++m)
        for (int part = 0; part < 2; ++part) {
          if (part && m == 0) continue;
          T t = {};
          t.g = make_int4(st, l, m, part);
          t.t.dst = (uint16_t)(part * nd + tri(l, m));
          t.t.flag = (uint8_t)((l & 1) | (part << 1));
          if (st == 1) {           // sum over source degrees n = m .. p-1
            if (m >= p) continue;
            t.t.cnt = (uint8_t)(p - m);
            t.t.src = (uint16_t)(part * ns + tri(m, m));
            t.t.step = (uint8_t)(m + 1);
          } else {                 // sum over source orders part .. l
            t.t.cnt = (uint8_t)(l + 1 - part);
            t.t.src = (uint16_t)(part * ns + tri(l, part));
            t.t.step = 1;
          }
          v.push_back(t);
        }
    std::stable_sort(v.begin(), v.end(),
                     [](const T &a, const T &b) { return a.t.cnt > b.t.cnt; });
    h.d.first[st] = (int)h.trip.size();
    h.d.rounds[st] = ((int)v.size() + 31) / 32;
    h.d.off[st] = off;
    for (int r = 0; r < h.d.rounds[st]; ++r) {
      h.trip.push_back(v[32 * r].t.cnt);
      h.toff.push_back(off);
      off += 32 * v[32 * r].t.cnt;
      for (int k = 0; k < 32; ++k) {
        T t = {};
        t.t.dst = 0xffff;
        t.g = make_int4(-1, 0, 0, 0);
        if (32 * r + k < (int)v.size()) t = v[32 * r + k];
        h.task.push_back(t.t);
        h.gen.push_back(t.g);
      }
    }
  }
  h.d.stride = off;
  return h;
}

// the units: child 0's offsets (dx, dy, dz) in [-3, 2]^3 minus [-1, 1]^3, one of
// each opposite pair; cell digits d + 3 in bits 0-2, 3-5, 6-8, bit 9 a pair,
// offset code of the direction tables from bit 16
std::vector<unsigned> make_units() {
  std::vector<unsigned> u;
  for (int c = 0; c < 6; ++c)
    for (int b = 0; b < 6; ++b)
      for (int a = 0; a < 6; ++a) {
        auto in = [](int v) { return v >= 2 && v <= 4; };
        if (in(a) && in(b) && in(c)) continue;
        const bool pair = a >= 1 && b >= 1 && c >= 1;      // -d is an offset too
        const int me = a + 6 * b + 36 * c, op = (6 - a) + 6 * (6 - b) + 36 * (6 - c);
        if (pair && op < me) continue;
        u.push_back((unsigned)(a | b << 3 | c << 6 | (pair ? 512 : 0) |
                               (unsigned)(a + 7 * b + 49 * c) << 16));
      }
  return u;
}

// a unit's stream table from its direction table (tables.cu, kind 0)
__global__ void k_m2l_fp64_tables(int p, int rounds, const unsigned *__restrict__ units,
                                  const int *__restrict__ trip, const int *__restrict__ toff,
                                  const int4 *__restrict__ gen, const double *__restrict__ dir,
                                  int ef, int ei, int vv, int dstride, int stride,
                                  double *__restrict__ out) {
  const int nm = tri(p), nl = tri(p + 1);
  const double *s = dir + (size_t)(units[blockIdx.x] >> 16) * dstride;
  double *o = out + (size_t)blockIdx.x * stride;
  for (int r = threadIdx.x >> 5; r < rounds; r += blockDim.x >> 5) {
    const int lane = threadIdx.x & 31;
    const int4 g = gen[32 * r + lane];
    for (int k = 0; k < trip[r]; ++k) {
      double v = 0.;
      if (g.x == 1) {              // order m, degree j, source degree n
        const int m = g.z, n = m + k, j = g.y;
        if (n < p) v = s[vv + m2l_vrow_off(p, n) + m * (p + 1) - m * (m - 1) / 2 + (j - m)];
      } else if (g.x >= 0) {
        const int m = g.w + k, nc = g.x == 0 ? nm : nl;
        if (m <= g.y)
          v = s[(g.x == 0 ? ef : ei) + 2 * (m2l_plane_off(nc, m) + tri(g.y, g.z) - tri(m)) + g.w];
      }
      o[toff[r] + 32 * k + lane] = v;
    }
  }
}

__device__ __forceinline__ double flip(double v, bool neg) {
  return __hiloint2double(__double2hiint(v) ^ (neg ? 0x80000000 : 0), __double2loint(v));
}

// sources of a unit: singly; in pairs, u and w made one after the other from
// sources read twice; in pairs, both made at once
enum { kF64Single = 0, kF64PairTwice = 1, kF64Pair = 2 };

// shared memory of a warp's sources, and of a warp, in doubles
__host__ __device__ inline int m2l_fp64_a(int p, int mode) {
  const int nm = tri(p), nl = tri(p + 1);
  return mode == kF64Pair && 4 * nm > 2 * nl ? 4 * nm : 2 * nl;
}
__host__ __device__ inline int m2l_fp64_warp(int p, int mode) {
  const int nm = tri(p), nl = tri(p + 1);
  return m2l_fp64_a(p, mode) + (mode != kF64Single && 4 * nm > 2 * nl ? 4 * nm : 2 * nl);
}

// R rounds of 32 lanes over the tri(p+1) local coefficients.  WHOLE: a CTA takes all
// segments, adding them up in the locals; else segment blockIdx.y
template <int R, bool WHOLE>
__global__ void __launch_bounds__(32 * kF64Warps, R <= 5 ? 3 : 2)
    k_m2l_fp64(int nparents, int nunits, int mode, const int *__restrict__ parents,
               const int *__restrict__ child, const int *__restrict__ begin,
               const int *__restrict__ end, const int *__restrict__ col,
               const int *__restrict__ ncol, const int *__restrict__ ijk,
               const uint8_t *__restrict__ depth, int p, M2lFp64Sched S,
               const F64Task *__restrict__ task, const int *__restrict__ trip,
               const unsigned *__restrict__ units, const double *__restrict__ tabs,
               const double *__restrict__ dir, int dstride, int ph_off,
               const uint8_t *__restrict__ lm, double scale_e,
               const cplx<double> *__restrict__ mult, cplx<double> *__restrict__ loc,
               cplx<double> *__restrict__ parts, uint8_t *__restrict__ marks) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int grid[216];
  const int nm = tri(p), nl = tri(p + 1);
  // a CTA takes all eight children of a parent, or half of them
  const int lane = threadIdx.x & 31, cw = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int halves = kF64Warps / nw, pb = blockIdx.x / halves;
  const int w = (blockIdx.x - pb * halves) * nw + cw;
  // per warp: A holds the phased sources (u and w, or u, then w), later z; B the
  // rotated ones (u and w), later the local: real plane, imaginary plane each
  double *A = reinterpret_cast<double *>(smem_raw) + (size_t)cw * m2l_fp64_warp(p, mode);
  double *B = A + m2l_fp64_a(p, mode);
  for (int i = threadIdx.x; i < 216; i += blockDim.x) grid[i] = -1;
  __syncthreads();
  const int P = parents[pb];
  {
    const int pi = ijk[3 * P], pj = ijk[3 * P + 1], pk = ijk[3 * P + 2];
    const int nc = ncol[P];
    for (int e = threadIdx.x; e < nc * 8; e += blockDim.x) {
      const int q = col[27 * P + e / 8];
      const int qc = child[q];
      if (qc < 0) continue;
      const int o = e & 7;
      const int s = qc + o;
      if (end[s] == begin[s]) continue;
      const int gx = 2 * (ijk[3 * q] - pi + 1) + (o & 1);
      const int gy = 2 * (ijk[3 * q + 1] - pj + 1) + ((o >> 1) & 1);
      const int gz = 2 * (ijk[3 * q + 2] - pk + 1) + ((o >> 2) & 1);
      grid[gx + 6 * (gy + 6 * gz)] = s;
    }
  }
  __syncthreads();
  const int t = child[P] + w;
  if (end[t] <= begin[t]) return;
  const int bx = w & 1, by = (w >> 1) & 1, bz = (w >> 2) & 1;
  // source at child 0's offset with cell digits a, b, c (see m2l_lanes.cuh)
  auto source_of = [&](int a, int b, int c) -> int {
    return grid[(bx ? a : 5 - a) + 6 * (by ? b : 5 - b) + 36 * (bz ? c : 5 - c)];
  };
  cplx<double> acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = cmake(0., 0.);
  bool any = false;                        // the segment has a source
  // a segment's sum: onto the local, zero before the pass (up to order 6 kept in
  // registers: one round), or to its place in the workspace with a mark that it is
  // there
  const double ih = ldexp(1.0, depth[t]) / scale_e;
  cplx<double> total = cmake(0., 0.);
  auto finish = [&](int seg) {
    const size_t at = ((size_t)seg * nparents + pb) * kF64Warps + w;
    if (!WHOLE && lane == 0) marks[at] = any;
    if (!any) return;
    cplx<double> *out = WHOLE ? loc + (size_t)t * nl : parts + at * nl;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = lane + 32 * r;
      if (k < nl) {
        const int l = lm[2 * k], m = lm[2 * k + 1];
        const bool sg = ((bz & (l + m)) ^ (bx & m)) & 1, cj = bx ^ by;
        const cplx<double> v = cmake(flip(acc[r].re * ih, sg), flip(acc[r].im * ih, sg ^ cj));
        if (WHOLE && R == 1) total = cadd(total, v);
        else out[k] = WHOLE ? cadd(out[k], v) : v;
        if (WHOLE) acc[r] = cmake(0., 0.);
      }
    }
    any = false;
  };
  int seg = WHOLE ? 0 : blockIdx.y, u = seg_unit(seg, nunits);
  int next = seg_unit(seg + 1, nunits);
  for (;; ++u) {
    if (u == next) {
      finish(seg);
      if (!WHOLE || ++seg == kF64Segs) break;
      next = seg_unit(seg + 1, nunits);
    }
    const unsigned code = units[u];
    const int a = code & 7, b = (code >> 3) & 7, c = (code >> 6) & 7;
    int s0 = source_of(a, b, c), s1 = (code & 512u) ? source_of(6 - a, 6 - b, 6 - c) : -1;
    if (s0 < 0 && s1 < 0) continue;
    any = true;
    // the opposite source alone: its terms with (-1)^l, odd degrees negated;
    // a pair taken singly: one after the other
    const bool both = s0 >= 0 && s1 >= 0;
    for (int turn = 0; turn < (both && mode == kF64Single ? 2 : 1); ++turn) {
      const bool two = both && mode != kF64Single;
      const bool opp = both ? turn == 1 : s0 < 0;
      const int sa = opp ? s1 : s0;
      const double *ph = dir + (size_t)(code >> 16) * dstride + ph_off;
      const double *tab = tabs + (size_t)u * S.stride + lane;
      // mirror S and z-phase of the sources: u = y + (-1)^l y' (or the one
      // source there is), w = y - (-1)^l y'
      auto load = [&](bool diff) {
        for (int k = lane; k < nm; k += 32) {
          const int l = lm[2 * k], m = lm[2 * k + 1];
          const bool sg = ((bz & (l + m)) ^ (bx & m)) & 1, cj = bx ^ by, odd = l & 1;
          const double cr = ph[2 * m], ci = ph[2 * m + 1];
          cplx<double> v = mult[(size_t)sa * nm + k];
          v.re = flip(v.re, sg ^ (opp && odd));
          v.im = flip(v.im, sg ^ cj ^ (opp && odd));
          if (two) {
            cplx<double> x = mult[(size_t)s1 * nm + k];
            x.re = flip(x.re, sg ^ odd);
            x.im = flip(x.im, sg ^ cj ^ odd);
            const cplx<double> d = cmake(v.re - x.re, v.im - x.im);
            v = diff ? d : cadd(v, x);
            if (mode == kF64Pair) {
              A[2 * nm + k] = d.re * cr - d.im * ci;
              A[3 * nm + k] = d.re * ci + d.im * cr;
            }
          }
          A[k] = v.re * cr - v.im * ci;
          A[nm + k] = v.re * ci + v.im * cr;
        }
        __syncwarp();
      };
      // one stage: every lane its dot product of each round
      auto stage = [&](int st, const double *in, int last, auto &&put) {
        const F64Task *tk = task + 32 * S.first[st] + lane;
        const int *tr = trip + S.first[st];
        const double *f = tab + S.off[st];
        for (int r = 0; r < S.rounds[st]; ++r, tk += 32) {
          const F64Task q = *tk;
          const int T = tr[r];
          int step = q.step;
          const double *x = in + q.src;
          if (st == 1 && two && (q.flag & 1)) x += 2 * nm;      // odd degrees from w
          double v = 0.;
          if (R > 8) {
            // few warps (order 22 and above): the loads of four steps ahead of their
            // products (past a product's end they read on, inside the vector and
            // the table, and count as zero).  60k Plummer particles, order 26 70 ms,
            // 72 without, order 29 130, 148; order 12, whose warps hide the loads,
            // 147 ms, 129 without
            int at = (int)(x - in);
            for (int k = 0; k < T; k += 4) {
              double e4[4], x4[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                e4[i] = __ldg(f + 32 * (k + i));
                x4[i] = in[min(at, last)];
                at += step;
                if (st == 1) ++step;
              }
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (k + i < T) v = fma(e4[i], k + i < q.cnt ? x4[i] : 0., v);
            }
            f += 32 * T;
          } else {
#pragma unroll 4
            for (int k = 0; k < T; ++k, f += 32) {
              const double e = __ldg(f);
              if (k < q.cnt) {
                v = fma(e, *x, v);
                x += step;
                if (st == 1) ++step;
              }
            }
          }
          if (q.dst != 0xffff) put(q, v);
        }
      };
      load(false);
      stage(0, A, 2 * nm - 1, [&](const F64Task &q, double v) { B[q.dst] = v; });
      if (two) {
        const bool again = mode == kF64PairTwice;
        __syncwarp();
        if (again) load(true);
        stage(0, again ? A : A + 2 * nm, 2 * nm - 1,
              [&](const F64Task &q, double v) { B[2 * nm + q.dst] = v; });
      }
      __syncwarp();
      // (no source term has order p: its place in z, the last of either plane)
      if (lane < 2) A[lane * nl + nl - 1] = 0.;
      stage(1, B, (two ? 4 : 2) * nm - 1, [&](const F64Task &q, double v) { A[q.dst] = flip(v, opp && (q.flag & 1)); });
      __syncwarp();
      stage(2, A, 2 * nl - 1, [&](const F64Task &q, double v) { B[q.dst] = v; });
      __syncwarp();
      // conjugate z-phase
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = lane + 32 * r;
        if (k < nl) {
          const int m = lm[2 * k + 1];
          const double cr = ph[2 * m], ci = ph[2 * m + 1];
          const double re = B[k], im = m ? B[nl + k] : 0.;
          acc[r].re = fma(re, cr, fma(im, ci, acc[r].re));
          acc[r].im = fma(im, cr, fma(-re, ci, acc[r].im));
        }
      }
      __syncwarp();
    }
  }
  if (WHOLE && R == 1 && lane < nl) loc[(size_t)t * nl + lane] = total;
}

// the segments added in order onto the locals (zero before the pass), one warp per
// child
__global__ void __launch_bounds__(32 * kF64Warps)
    k_m2l_parts_sum(int nparents, const int *__restrict__ parents, const int *__restrict__ child,
                    const int *__restrict__ begin, const int *__restrict__ end, int nl,
                    const cplx<double> *__restrict__ parts, const uint8_t *__restrict__ marks,
                    cplx<double> *__restrict__ loc) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int t = child[parents[blockIdx.x]] + w;
  if (end[t] <= begin[t]) return;
  const size_t step = (size_t)nparents * kF64Warps, at = (size_t)blockIdx.x * kF64Warps + w;
  const bool there = lane < kF64Segs && marks[lane < kF64Segs ? lane * step + at : 0];
  const unsigned segs = __ballot_sync(0xffffffffu, there);
  if (segs == 0) return;
  for (int c = lane; c < nl; c += 32) {
    cplx<double> v = loc[(size_t)t * nl + c];
    for (unsigned m = segs; m; m &= m - 1)
      v = cadd(v, parts[((__ffs(m) - 1) * step + at) * nl + c]);
    loc[(size_t)t * nl + c] = v;
  }
}

}  // namespace

void build_m2l_fp64_tables(OpTables<double> &tb, cudaStream_t st) {
  const int p = tb.p;
  const HostSched h = make_sched(p);
  const std::vector<unsigned> units = make_units();
  const size_t nr = h.trip.size(), nt = h.task.size();
  M2lFp64Tables &f = tb.m2l64;
  f.nunits = (int)units.size();
  f.sched = h.d;
  f.tabs.reserve((size_t)h.d.stride * units.size() + 4 * 32);   // read on by up to 3 steps
  f.task.reserve(nt);
  f.trip.reserve(nr);
  f.units.reserve(units.size());
  DBuf<int> toff;
  DBuf<int4> gen;
  toff.reserve(nr);
  gen.reserve(nt);
  static_assert(sizeof(F64Task) == sizeof(uint64_t), "tasks are kept as 64-bit words");
  ACHECK(cudaMemcpyAsync(f.task.ptr, h.task.data(), nt * sizeof(F64Task), cudaMemcpyHostToDevice, st));
  ACHECK(cudaMemcpyAsync(f.trip.ptr, h.trip.data(), nr * sizeof(int), cudaMemcpyHostToDevice, st));
  ACHECK(cudaMemcpyAsync(toff.ptr, h.toff.data(), nr * sizeof(int), cudaMemcpyHostToDevice, st));
  ACHECK(cudaMemcpyAsync(gen.ptr, h.gen.data(), nt * sizeof(int4), cudaMemcpyHostToDevice, st));
  ACHECK(cudaMemcpyAsync(f.units.ptr, units.data(), units.size() * sizeof(unsigned),
                         cudaMemcpyHostToDevice, st));
  k_m2l_fp64_tables<<<(int)units.size(), 256, 0, st>>>(
      p, (int)nr, f.units.ptr, f.trip.ptr, toff.ptr, gen.ptr, tb.dir_m2l.ptr, dir_offset(p, 0, 0),
      dir_offset(p, 0, 2), dir_offset(p, 0, 7), dir_offset(p, 0, 6), h.d.stride, f.tabs.ptr);
  ACHECK(cudaGetLastError());
  ACHECK(cudaStreamSynchronize(st));
  toff.release();
  gen.release();
}

void launch_m2l_fp64(AranGpuSolver3d *s, const int *parents, int count, cudaStream_t st) {
  if (count <= 0) return;
  DevTree &t = s->tree;
  OpTables<double> &tb = s->t64;
  const M2lFp64Tables &f = tb.m2l64;
  const int p = s->cfg.order, nm = tri(p), nl = tri(p + 1);
  int dev_smem = 0, sm_smem = 0, nsm = 0;
  ACHECK(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
  ACHECK(cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, s->device));
  ACHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, s->device));
  // Pairs, made at once (16 warps an SM or more up to order 20); read twice where
  // that keeps 16 warps (orders 21 to 23): order 22, 60k Plummer particles, M2L 44
  // ms, 71 made at once, 50 singly; 2 to 3 % slower below.  Above, read twice by
  // CTAs of four warps where those make 12 (orders 24 to 27): order 26, 72 ms, 76 singly;
  // singly where that leaves 16 warps and pairs 8 (order 28); order 29 (8 either
  // way) 148 ms in pairs, 170 singly.
  auto bytes = [&](int nw, int mode) { return (size_t)nw * m2l_fp64_warp(p, mode) * sizeof(double); };
  auto warps = [&](int nw, int mode) {
    return bytes(nw, mode) + 1024 > (size_t)dev_smem
               ? 0
               : std::min(16, nw * (int)(sm_smem / (bytes(nw, mode) + 2048)));
  };
  int nw = kF64Warps, mode = kF64Pair;
  if (warps(nw, kF64PairTwice) > warps(nw, mode)) mode = kF64PairTwice;
  if (warps(nw, mode) < 12 && warps(4, kF64PairTwice) >= 12) {
    nw = 4;
    mode = kF64PairTwice;
  } else if (warps(nw, kF64Single) > warps(nw, mode)) {
    mode = kF64Single;
  }
  const size_t sm = bytes(nw, mode);
  // A CTA per segment where one per parent would leave the last wave of CTAs a large
  // part of the pass: 176 parents of order 12 1.28 ms, 3.1 with a CTA for all
  // segments, 1,574 14.3 and 16.1, 3,941 36.7 and 37.6; forests of small systems,
  // whose parents have few sources for a CTA's set-up, the other way about from fewer
  // on: 2,500 parents in 300 systems, order 16, 24.9 and 19.3 ms, 21,600 in
  // 300 319 and 291, 2,880 in 40 42.6 either way, 335 in 40 3.5 either way.
  const bool whole = count > 24 * nsm || (count > 8 * nsm && count < 32 * (int64_t)s->nsys);
  const size_t per = (size_t)kF64Segs * kF64Warps;         // segments' sums of a parent
  int step = count;
  cplx<double> *parts = nullptr;
  uint8_t *marks = nullptr;
  if (!whole) {
    // as many parents at a time as the workspace holds
    const int most = (int)(kM2lFp64PartBytes / (int64_t)(per * nl * sizeof(cplx<double>)));
    step = ceil_div(count, ceil_div(count, most));
    s->m2l_part64.reserve(per * step * (2 * nl + 1));
    parts = reinterpret_cast<cplx<double> *>(s->m2l_part64.ptr);
    marks = reinterpret_cast<uint8_t *>(parts + per * step * nl);
  }
  const cplx<double> *mult = reinterpret_cast<cplx<double> *>(s->mult64.ptr);
  cplx<double> *loc = reinterpret_cast<cplx<double> *>(s->loc64.ptr);
  auto run = [&](auto kern) {
    smem_opt_in(kern, sm);
    for (int first = 0; first < count; first += step) {
      const int cnt = std::min(step, count - first);
      kern<<<dim3(cnt * (kF64Warps / nw), whole ? 1 : kF64Segs), 32 * nw, sm, st>>>(
          cnt, f.nunits, mode, parents + first, t.child.ptr, t.begin.ptr, t.end.ptr, t.col.ptr,
          t.ncol.ptr, t.ijk.ptr, t.depth.ptr, p, f.sched,
          reinterpret_cast<const F64Task *>(f.task.ptr), f.trip.ptr, f.units.ptr, f.tabs.ptr,
          tb.dir_m2l.ptr, dir_offset(p, 0, 6), dir_offset(p, 0, 4), tb.lm.ptr, s->scale_e, mult,
          loc, parts, marks);
      ACHECK(cudaGetLastError());
      s->launches++;
      if (!whole) {
        k_m2l_parts_sum<<<cnt, 32 * kF64Warps, 0, st>>>(cnt, parents + first, t.child.ptr,
                                                        t.begin.ptr, t.end.ptr, nl, parts, marks,
                                                        loc);
        ACHECK(cudaGetLastError());
        s->launches++;
      }
    }
  };
  auto pick = [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    if (whole) run(k_m2l_fp64<R, true>);
    else run(k_m2l_fp64<R, false>);
  };
  if (nl <= 32) pick(std::integral_constant<int, 1>{});
  else if (nl <= 96) pick(std::integral_constant<int, 3>{});
  else if (nl <= 160) pick(std::integral_constant<int, 5>{});
  else if (nl <= 256) pick(std::integral_constant<int, 8>{});
  else pick(std::integral_constant<int, 16>{});
}

}  // namespace aran
