// leaf_fp64.cu -- P2M and L2P in FP64 (up_func's and down_func's leaf parts:
// aran/arandevelopment3d.c:169-216 and :285-356).  The FP64 pipe takes half a
// lane per cycle and scheduler, so its instructions times the lanes they leave
// idle are the whole cost; shared memory and index arithmetic come free.
#include "internal.cuh"

namespace aran {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 4;

__device__ __forceinline__ double leaf_inv_scale(int depth, double scale_e) {
  return ldexp(1.0, depth) / scale_e;    // 1/h_d = 2^d / 2^E (exact power of two)
}

// P2M.  A leaf's particles are taken in segments of 32 from its first on, and a
// leaf's sum is the sum of its segments in order (k_p2m64_sum), each added up
// particle by particle: what else is solved, and with it the leaf's place among the
// sorted particles, does not change its bits.  A warp takes the segments that start
// in its span of places, 32 particles at a time whatever segments they lie in (a
// warp per leaf keeps as many lanes busy as the leaf has points).  A lane makes
// its particle's q S_l^m in m-major order (six operations a coefficient) into
// shared memory; every 32 values the lanes turn to the values, a lane one of them,
// and add it up (one addition a value and particle; by shuffles over the warp it was
// five on every lane).  The first segment of a leaf goes to its multipole, the
// others to a workspace, at the window of 32 places in which they start: no two start
// in one.  With few segments (segs > 0) a warp takes one, segment u mod segs of leaf
// u / segs: fewer rounds in turn, and few CTAs, which stay clear of the near
// field's.  Order 12, Plummer particles: 200k (18 a leaf) 0.43 ms, 0.48 with spans of 32,
// 1.44 with a warp per leaf and shuffles (0.34 with parts of leaves added as they come;
// the solve 38.1 ms either way); 4M 7.1 and 8.2 ms; 3k 0.045 ms.
constexpr int kFewSegs = 4096;

__global__ void __launch_bounds__(32 * kWarps)
    k_p2m64(int64_t n, int nleaves, int segs, int span,
            const int *__restrict__ win_leaf,
            const int2 *__restrict__ leaf_be, const int *__restrict__ leaf_node,
            const uint8_t *__restrict__ depth, const real4<double> *__restrict__ rel, int p,
            const double *__restrict__ rec_g, const double *__restrict__ p2mf_g, double scale_e,
            double *__restrict__ mult, double *__restrict__ more) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nm = tri(p);
  double *rec = reinterpret_cast<double *>(smem_raw);   // (c0, c1) by (l, m)
  double *fac = rec + 2 * nm;                            // by m-major place
  int *coef = reinterpret_cast<int *>(fac + nm);         // (l, m) of a place
  double *buf = reinterpret_cast<double *>(coef + ((nm + 1) & ~1));
  for (int i = threadIdx.x; i < 2 * nm; i += blockDim.x) rec[i] = rec_g[i];
  for (int i = threadIdx.x; i < nm; i += blockDim.x) {
    int l, m;
    mmajor_lm(i, p - 1, l, m);
    fac[i] = p2mf_g[l];
    coef[i] = tri(l, m);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  buf += w * (32 * 33 + 2 * nm);
  double *carry = buf + 32 * 33;           // sums of a segment that goes on
  // first segment that starts at or behind a place: its leaf and its own place (the
  // whole warp asks)
  auto segment_from = [&](int64_t at, int &leaf) -> int {
    leaf = nleaves;
    if (at >= n) return (int)n;
    const int L = win_leaf[at >> 5];     // of the place's window of 32
    leaf = L + __popc(__ballot_sync(kFull, L + lane < nleaves &&
                                               leaf_be[min(L + lane, nleaves - 1)].x < at));
    if (leaf > L) {                      // the place may lie inside the leaf before
      const int2 be = leaf_be[leaf - 1];
      const int64_t next = be.x + ((at - be.x + 31) & ~(int64_t)31);
      if (next < be.y) {
        --leaf;
        return (int)next;
      }
    }
    return leaf < nleaves ? leaf_be[leaf].x : (int)n;
  };
  const int64_t u = blockIdx.x * (int64_t)kWarps + w;
  int L0, base, stop;                      // L0: leaf of the round's first particle
  if (segs > 0) {
    L0 = (int)(u / segs);
    if (L0 >= nleaves) return;
    const int2 be = leaf_be[L0];
    base = be.x + 32 * (int)(u - (int64_t)L0 * segs);
    stop = min(base + 32, be.y);
  } else {
    int L1;
    base = segment_from(span * u, L0);
    stop = segment_from(span * (u + 1), L1);
  }
  bool goes_on = false;                    // its segment began in a round before
  for (; base < stop; base += 32) {
    const int cnt = min(stop - base, 32);
    // bit i: particle base + i starts a leaf, a segment (never the first)
    unsigned bit = 0;
    if (lane > 0 && L0 + lane < nleaves) {
      const int at = leaf_be[L0 + lane].x - base;
      if (at < cnt) bit = 1u << at;
    }
    const unsigned starts = __reduce_or_sync(kFull, bit);
    const int L = L0 + __popc(starts & ((2u << lane) - 1u));
    const unsigned cuts =
        __ballot_sync(kFull, lane > 0 && lane < cnt && ((base + lane - leaf_be[L].x) & 31) == 0);
    double x = 0, y = 0, z = 0, q = 0;
    if (lane < cnt) {
      const double ih = leaf_inv_scale(depth[leaf_node[L]], scale_e);
      const real4<double> r = rel[base + lane];
      x = r.x * ih;
      y = r.y * ih;
      z = r.z * ih;
      q = r.q;
    }
    const double r2 = x * x + y * y + z * z;
    int k = 0;                               // value: 2 m-major place + part
    auto put = [&](double v) {
      buf[(k & 31) * 33 + lane] = v;
      ++k;
      if ((k & 31) && k < 2 * nm) return;
      // the lanes take the values
      __syncwarp();
      const int mine = ((k - 1) & ~31) + lane;
      if (mine < k) {
        const double f = (mine & 1) ? -fac[mine >> 1] : fac[mine >> 1];
        const size_t c = 2 * (size_t)coef[mine >> 1] + (mine & 1);
        double sum = goes_on ? carry[mine] : 0.;
        unsigned left = cuts;
        int l = L0, j = 0;
        while (j < cnt) {
          const int j1 = left ? __ffs(left) - 1 : cnt;
          left &= left - 1;
#pragma unroll 4
          for (int jj = j; jj < j1; ++jj) sum += buf[lane * 33 + jj];
          j = j1;
          const int2 be = leaf_be[l];
          const bool last = base + j == be.y;
          if (last || ((base + j - be.x) & 31) == 0) {   // a segment ends
            const int k0 = (base + j - 1 - be.x) & ~31;    // its place in the leaf
            double *out = k0 == 0 ? mult + 2 * (size_t)nm * leaf_node[l]
                                  : more + 2 * (size_t)nm * ((be.x + k0) >> 5);
            out[c] = f * sum;
            sum = 0.;
            if (last) ++l;
          }
        }
        carry[mine] = sum;
      }
      __syncwarp();
    };
    double dre = q * rec[0], dim = 0;
    for (int m = 0; m < p; ++m) {
      if (m > 0) {
        const double a = rec[2 * tri(m, m)];
        const double nre = a * (x * dre - y * dim), nim = a * (x * dim + y * dre);
        dre = nre;
        dim = nim;
      }
      double s1re = dre, s1im = dim, s2re = 0, s2im = 0;
      put(dre);
      put(dim);
      for (int l = m + 1; l < p; ++l) {
        const double a = rec[2 * tri(l, m)] * z, b = rec[2 * tri(l, m) + 1] * r2;
        const double sre = a * s1re - b * s2re, sim = a * s1im - b * s2im;
        s2re = s1re;
        s2im = s1im;
        s1re = sre;
        s1im = sim;
        put(sre);
        put(sim);
      }
    }
    L0 += __popc(starts);
    const int2 be = leaf_be[L0];
    goes_on = ((base + cnt - be.x) & 31) != 0 && be.y != base + cnt;
    if (be.y == base + cnt) ++L0;
  }
}

// the segments of leaves of more than 32 particles in order, 32 threads per leaf, 128
// where there are many values
__global__ void __launch_bounds__(128)
    k_p2m64_sum(int nleaves, int per, const int2 *__restrict__ leaf_be,
                const int *__restrict__ leaf_node, int nv, const double *__restrict__ more,
                double *__restrict__ mult) {
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int L = (int)(g / per);
  if (L >= nleaves) return;
  const int2 be = leaf_be[L];
  if (be.y - be.x <= 32) return;
  double *out = mult + (size_t)nv * leaf_node[L];
  for (int c = (int)(g - (int64_t)L * per); c < nv; c += per) {
    double v = out[c];
    for (int at = be.x + 32; at < be.y; at += 32) v += more[(size_t)nv * (at >> 5) + c];
    out[c] = v;
  }
}

// L2P, a warp per leaf.  What a particle's solid harmonic S_l^m is multiplied
// with is made once per leaf: for the potential, the z derivative and the x and
// y derivatives (whose terms of orders m and -m fold into four real factors), so
// a particle takes 14 operations per (l, m) with the field, 23 before.  200k
// Plummer particles (18 a leaf), order 12, field: 0.96 ms, 1.73 before.
template <bool FIELD>
__global__ void __launch_bounds__(32 * kWarps)
    k_l2p64(int nleaves, const int *__restrict__ leaf_node, const int2 *__restrict__ leaf_be,
            const uint8_t *__restrict__ depth, const real4<double> *__restrict__ rel, int p,
            const double *__restrict__ rec_g, const double *__restrict__ gz_g,
            const double *__restrict__ gm_g, double scale_e, const cplx<double> *__restrict__ loc,
            double *__restrict__ acc_pot, double *__restrict__ acc_fld) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NF = FIELD ? 4 : 1;        // pairs of factors per (l, m)
  const int nl = tri(p + 1);
  double2 *rec = reinterpret_cast<double2 *>(smem_raw);
  for (int i = threadIdx.x; i < nl; i += blockDim.x)
    rec[i] = make_double2(rec_g[2 * i], rec_g[2 * i + 1]);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double2 *F = rec + nl + (size_t)w * nl * NF;
  const int L = blockIdx.x * kWarps + w;
  if (L >= nleaves) return;
  const int node = leaf_node[L];
  const cplx<double> *Lc = loc + (size_t)node * nl;
  for (int c = lane; c < nl; c += 32) {
    // degree of the triangular index c: floor((sqrt(8c+1)-1)/2), corrected
    int l = (int)((sqrtf(8.f * c + 1.f) - 1.f) * 0.5f);
    while (tri(l + 1) <= c) ++l;
    while (tri(l) > c) --l;
    const int m = c - tri(l);
    const double wm = m == 0 ? 1. : 2.;
    const cplx<double> v = Lc[c];
    F[c * NF] = make_double2(wm * v.re, -wm * v.im);
    if (FIELD && l < p) {
      const cplx<double> a = Lc[tri(l + 1, m)];
      const double g = wm * gz_g[c];
      F[c * NF + 1] = make_double2(a.re * g, -a.im * g);
      // terms of +m and, with S^{-m} = (-1)^m conj(S^m), of -m
      const double gp = gm_g[l * l + l + m];
      const cplx<double> bp = Lc[tri(l + 1, m + 1)];
      double rr = bp.re * gp, ri = -bp.im * gp, ii = bp.re * gp, ir = bp.im * gp;
      if (m > 0) {
        const double sg = (m & 1) ? -1. : 1., gn = gm_g[l * l + l - m];
        cplx<double> u = Lc[tri(l + 1, m - 1)];
        // L^{1-m} for m > 1
        if (m > 1) u = ((m - 1) & 1) ? cmake(-u.re, u.im) : cmake(u.re, -u.im);
        const double ur = sg * (u.re * gn), ui = sg * (u.im * gn);
        rr += ur;
        ri += ui;
        ii -= ur;
        ir += ui;
      }
      F[c * NF + 2] = make_double2(rr, ri);   // real part from S.re, S.im
      F[c * NF + 3] = make_double2(ir, ii);   // imaginary part
    }
  }
  __syncwarp();
  const int2 be = leaf_be[L];
  const double ih = leaf_inv_scale(depth[node], scale_e);
  for (int i = be.x + lane; i < be.y; i += 32) {
    const real4<double> r = rel[i];
    const double x = r.x * ih, y = r.y * ih, z = r.z * ih;
    const double r2 = x * x + y * y + z * z;
    double phi = 0, dz = 0, gre = 0, gim = 0;
    double dre = rec[0].x, dim = 0;
    auto add = [&](int c, bool grad, double sre, double sim) {
      const double2 f = F[c * NF];
      phi = fma(f.x, sre, fma(f.y, sim, phi));
      if (FIELD && grad) {
        const double2 a = F[c * NF + 1], g = F[c * NF + 2], h = F[c * NF + 3];
        dz = fma(a.x, sre, fma(a.y, sim, dz));
        gre = fma(g.x, sre, fma(g.y, sim, gre));
        gim = fma(h.x, sre, fma(h.y, sim, gim));
      }
    };
#pragma unroll 1
    for (int m = 0; m <= p; ++m) {
      if (m > 0) {
        const double a = rec[tri(m, m)].x;
        const double nre = a * (x * dre - y * dim), nim = a * (x * dim + y * dre);
        dre = nre;
        dim = nim;
      }
      double s1re = dre, s1im = dim, s2re = 0, s2im = 0;
      add(tri(m, m), m < p, dre, dim);
#pragma unroll 4
      for (int l = m + 1; l <= p; ++l) {
        const int c = tri(l, m);
        const double2 cc = rec[c];
        const double a = cc.x * z, b = cc.y * r2;
        const double sre = a * s1re - b * s2re, sim = a * s1im - b * s2im;
        s2re = s1re;
        s2im = s1im;
        s1re = sre;
        s1im = sim;
        add(c, l < p, sre, sim);
      }
    }
    acc_pot[i] += phi;
    if (FIELD) {
      acc_fld[3 * (size_t)i] += gre * ih;
      acc_fld[3 * (size_t)i + 1] += -gim * ih;
      acc_fld[3 * (size_t)i + 2] += dz * ih;
    }
  }
}

}  // namespace

void launch_p2m64(AranGpuSolver3d *s, cudaStream_t st) {
  DevTree &t = s->tree;
  OpTables<double> &tb = s->t64;
  const int p = s->cfg.order, nm = tri(p);
  const size_t sm = (size_t)3 * nm * sizeof(double) + ((nm + 1) & ~1) * sizeof(int) +
                    (size_t)kWarps * (32 * 33 + 2 * nm) * sizeof(double);
  smem_opt_in(k_p2m64, sm);
  s->m2l_part64.reserve(2 * (size_t)nm * ceil_div(t.n, 32));   // free until the M2L
  // few segments: a warp each, in few CTAs, which stay clear of the near field's
  const int per_leaf = ceil_div(t.max_leaf, 32);
  const bool few = t.nleaves * (int64_t)per_leaf <= kFewSegs;
  const int span = t.n < 150000 ? 32 : 128;   // 100k particles 0.28 ms, 0.29 with 128
  const int64_t warps = few ? t.nleaves * (int64_t)per_leaf : ceil_div(t.n, span);
  k_p2m64<<<ceil_div(warps, kWarps), 32 * kWarps, sm, st>>>(
      t.n, t.nleaves, few ? per_leaf : 0, span, t.win_leaf.ptr, t.leaf_be.ptr, t.leaf_node.ptr,
      t.depth.ptr, s->rel64.ptr, p, tb.rec.ptr, tb.p2mf.ptr, s->scale_e, s->mult64.ptr, s->m2l_part64.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  if (t.max_leaf > 32) {
    const int per = nm > 64 ? 128 : 32;
    k_p2m64_sum<<<ceil_div(t.nleaves * (int64_t)per, 128), 128, 0, st>>>(
        t.nleaves, per, t.leaf_be.ptr, t.leaf_node.ptr, 2 * nm, s->m2l_part64.ptr, s->mult64.ptr);
    ACHECK(cudaGetLastError());
    s->launches++;
  }
}

void launch_l2p64(AranGpuSolver3d *s, cudaStream_t st) {
  DevTree &t = s->tree;
  OpTables<double> &tb = s->t64;
  const int p = s->cfg.order, nl = tri(p + 1);
  const bool field = s->cfg.field != 0;
  const size_t sm = (size_t)nl * sizeof(double2) * (1 + kWarps * (field ? 4 : 1));
  auto kern = field ? k_l2p64<true> : k_l2p64<false>;
  smem_opt_in(kern, sm);
  kern<<<ceil_div(t.nleaves, kWarps), 32 * kWarps, sm, st>>>(
      t.nleaves, t.leaf_node.ptr, t.leaf_be.ptr, t.depth.ptr, s->rel64.ptr, p, tb.rec.ptr,
      tb.gz.ptr, tb.gm.ptr, s->scale_e, reinterpret_cast<const cplx<double> *>(s->loc64.ptr),
      s->acc_pot.ptr, s->acc_fld.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
}

}  // namespace aran
